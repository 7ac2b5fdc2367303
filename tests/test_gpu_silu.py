"""silu(gate) * up over every bf16 gate there is, the strongly negative ones among them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gates(device):
    return torch.arange(-32768, 32768, dtype=torch.int32, device=device).to(torch.int16).view(torch.bfloat16)


@pytest.mark.parametrize("up", [1.0, -0.7734375, 3.0e38, 2.0 ** -120])
def test_silu_mul_over_all_gates(capi, device, up):
    """The two roundings of F.silu(gate) * up on bf16 tensors; torch's silu divides in fp32 as the kernel's expression does."""
    gate = _gates(device).view(64, 1024)
    ups = torch.full_like(gate, up)
    got, want = capi.silu_mul(gate, ups), torch.nn.functional.silu(gate) * ups
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0))
    finite = torch.isfinite(gate)
    exact = gate.double() / (1.0 + torch.exp(-gate.double()))
    silu = capi.silu_mul(gate, torch.ones_like(gate)).double()
    # fp32: exp overflows below about -88.7, where the result is under 3e-37 in size; elsewhere half a unit of the last place of bf16
    # (2^-8) and the errors of fp32, 2^-21
    assert bool(((silu - exact).abs()[finite] <= (2.0 ** -8 + 2.0 ** -21) * exact.abs()[finite] + torch.where(gate.double()[finite] < -88.0, 3e-37, 1e-40)).all())


@pytest.mark.parametrize("limit", [0.0, 7.0])
@pytest.mark.parametrize("up", [1.0, -2.6875, 2.0 ** -100])
def test_gated_act_over_all_gates(pkg, device, up, limit):
    gate = _gates(device)[torch.isfinite(_gates(device))].view(-1, 255)
    ups = torch.full_like(gate, up)
    got = pkg.mixers.gated_act(torch.cat([gate, ups], dim=1), limit=limit).double()
    z, u, alpha = gate.double(), ups.double(), 1.0
    if limit:
        z, u, alpha = z.clamp(max=limit), u.clamp(-limit, limit) + 1.0, float(torch.tensor(1.702))
    want = z / (1.0 + torch.exp(-alpha * z)) * u
    # half a unit of bf16's last place (2^-8) and fp32's errors: of the exponent alpha z (up to 88.7) a unit of its last place, 2^-18, of the
    # rest 2^-21; where exp overflows (alpha z below about -88.7), up to 89 / 2^128 is lost; the smallest bf16 number is 9.2e-41
    bound = (2.0 ** -8 + 2.0 ** -18 + 2.0 ** -21) * want.abs() + 1e-40 + torch.where(alpha * z < -88.0, 3e-37 * u.abs(), 0.0)
    fits = want.abs() <= 3.38e38                                # the rest rounds to the largest or to infinity
    assert bool(((got - want).abs() <= bound)[fits].all()) and bool((fits | (got.abs() >= 3.38e38)).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,ff", [(1, 1), (1, 2048), (3, 1365), (511, 8), (513, 8), (2, 4104)])
def test_gated_act_at_the_edges_of_its_blocks(pkg, device, rows, ff, dtype):
    g = torch.Generator(device=device).manual_seed(rows + ff)
    gu = torch.randn(rows, 2 * ff, generator=g, device=device).to(dtype)
    z, u = gu.double()[:, :ff], gu.double()[:, ff:]
    want = z * torch.sigmoid(z) * u
    assert bool(((pkg.mixers.gated_act(gu).double() - want).abs() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21) * 1.01 * want.abs() + 1e-30).all())
