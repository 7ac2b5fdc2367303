"""Nucleus sampling by counts lists the nucleus' entries per warp, 512 places at a time, found by packed compares: against the form by
masses, bit for bit, for lists that overflow, ties across them, rows that end inside a lane's group of 16, and logits whose order a compare
could lose (zeros of both signs, subnormals)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
LONG = 8 * 8191 * 8 + 8      # one group more than eight CTAs count: by masses


@pytest.mark.parametrize("rows,vocab", [(3, 511), (3, 512), (75, 4097 + 15), (34, 2 * 32 * 512 + 1), (34, 2 * 32 * 2048 - 17), (5, 128256)])
@pytest.mark.parametrize("kind", ["dense", "subnormal", "two"])
@pytest.mark.parametrize("top_p", [0.5, 0.95, 1.0])
def test_lists_change_no_bit(capi, device, rows, vocab, kind, top_p):
    g = torch.Generator(device=device).manual_seed(rows + vocab)
    x = torch.randn(rows, vocab, generator=g, device=device)
    if kind == "dense":
        x = (x * 0.05).bfloat16()                       # half of the row and more is in the nucleus
    elif kind == "subnormal":
        x = (x * 3).round().to(torch.int16)             # patterns of zero and of the least subnormals, either sign
        x = torch.where(x < 0, x.abs() | -32768, x).view(torch.bfloat16)
        x[:, ::7] = -0.0
    else:
        x = (x > 0).bfloat16()                          # all ties
    long = torch.full((rows, LONG), float("-inf"), dtype=torch.bfloat16, device=device)
    long[:, :vocab] = x

    def run(logits):
        tokens, count = torch.zeros(rows, 1, dtype=torch.int64, device=device), torch.zeros(rows, dtype=torch.int32, device=device)
        mass, seen = torch.zeros(rows, device=device), []
        for seed in range(4):
            capi.top_p_step(logits, 0.9, top_p, seed, tokens, nucleus_count=count, nucleus_mass=mass)
            seen += [tokens.clone(), count.clone(), mass.clone()]
        return seen

    if top_p == 1.0:                                    # (the tail's entries without mass count as the nucleus' too)
        pairs = [(a, b) for i, (a, b) in enumerate(zip(run(x), run(long))) if i % 3 != 1]
    else:
        pairs = zip(run(x), run(long))
    for a, b in pairs:
        assert torch.equal(a, b)
