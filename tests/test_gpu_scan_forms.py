"""Recurrent scans of as many heads as take each form of the scan (columns per warp, warps per CTA, CTAs per SM), against the same
sequences one at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,H,D,batch", [("delta", 16, 128, 3), ("delta", 16, 128, 5), ("delta", 16, 128, 6), ("delta", 15, 120, 7),
                                            ("mix", 32, 64, 3), ("mix", 32, 64, 5), ("delta", 2, 128, 1), ("mix", 3, 4, 2)])
def test_forms_agree(pkg, device, kind, H, D, batch):
    from importlib import import_module

    mixers = import_module(pkg.__name__ + ".mixers")
    T = 37
    g = torch.Generator(device=device).manual_seed(H + D + batch)

    def rand(*shape, dtype=torch.float32):
        return torch.randn(*shape, generator=g, device=device).to(dtype)

    dt = torch.float32 if kind == "delta" else torch.bfloat16
    q, k = (rand(batch, T, H, D).mul_(D ** -0.5).to(dt) for _ in range(2))
    v, gate = (rand(batch, T, H, D, dtype=torch.bfloat16) for _ in range(2))
    decay = torch.rand(batch, T, H, D, generator=g, device=device).to(dt)
    state, positions, norm = rand(batch, H, D, D), torch.ones(batch, dtype=torch.int32, device=device), torch.ones(D, device=device)
    beta, bonus, bias = torch.rand(batch, T, H, generator=g, device=device), rand(H, D), rand(H * D) - 2.0

    def run(rows):
        s = state[rows].clone()
        extra = dict(beta=beta[rows].contiguous()) if kind == "delta" else dict(bonus=bonus, g_bias=bias)
        out = mixers.recurrent_scan(q[rows].contiguous(), k[rows].contiguous(), v[rows].contiguous(), decay[rows].contiguous(), s, positions[rows],
                                    norm, gate[rows].contiguous(), act=0, eps=1e-5, **extra)
        return out.float(), s

    got, want = run(slice(0, batch)), [run(slice(b, b + 1)) for b in range(batch)]
    for b in range(batch):
        # sums of up to 128 fp32 products in another order, carried through 37 tokens: far below 1e-4 of the result
        assert float((got[1][b] - want[b][1][0]).norm() / want[b][1][0].norm()) < 1e-4
        # bf16 outputs, normed: half a unit in the last place on either side
        assert float((got[0][b] - want[b][0][0]).norm() / want[b][0][0].norm()) < 2.0 ** -8


@pytest.mark.parametrize("batch", [3, 5, 6, 12])
@pytest.mark.parametrize("D", [32, 64])
def test_forms_of_the_delta_rule_with_few_rows(pkg, device, D, batch):
    test_forms_agree(pkg, device, "delta", 16, D, batch)
