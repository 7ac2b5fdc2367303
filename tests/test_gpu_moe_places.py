"""Experts of few tokens as groups of products over places by expert (`l3ci_moe_gather_places`, `l3ci_linear_gated`): places without a pair,
every width of the products' narrow side, tiles that end inside, and a limit of the gates, against the float64 restatement."""
import ctypes as C

import pytest
import torch

from oracle import rupotar as ref

pytestmark = pytest.mark.gpu


def rand(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16()


@pytest.mark.parametrize("rows", [1, 8, 9, 17, 32])
@pytest.mark.parametrize("E,top,width,ff", [(4, 4, 64, 40), (7, 2, 72, 136), (1, 1, 2048, 64)])
def test_experts_of_few_tokens(pkg, device, rows, E, top, width, ff):
    mx, limit = pkg.mixers, 0.7
    h, z = rand(rows, width, seed=1), rand(rows, E, seed=2, scale=5).float()
    gate, up, down = (rand(E, *s, seed=i, scale=s[1] ** -0.5) for i, s in enumerate(((ff, width), (ff, width), (width, ff)), 3))
    experts, ranks, weights, counts = mx.moe_route(z.to(device), torch.zeros(E, device=device), top)
    x, part_rows = mx.moe_places(h.to(device), experts, ranks, E)
    e, at = experts.cpu().long(), part_rows.cpu().long()
    assert torch.equal(at, e * rows + ranks.cpu()) and at.unique().numel() == rows * top
    assert torch.equal(x.flatten(0, 1)[at.flatten().to(device)].cpu(), h.repeat_interleave(top, 0))
    for early in (False, True):
        a = mx.few_rows(x, torch.cat([gate, up], 1).to(device), mx.ACT_SILU_GATE, early=early, always=True, limit=limit, alpha=1.702)
        y = mx.few_rows(a, down.to(device), early=early, always=True)
        stream = torch.zeros(rows, width, device=device)
        mx.residual_norm(y, stream, dtype=torch.bfloat16, part_rows=part_rows, part_weights=weights)
        want = torch.zeros(rows, width, dtype=torch.float64)
        for t in range(rows):
            for k in range(top):
                n = e[t, k]
                want[t] += weights.cpu().double()[t, k] * ref.clamped_expert(gate[n].double(), up[n].double(), down[n].double(), h[t].double(), limit)
        rel = (stream.double().cpu() - want).norm(dim=-1) / (want.norm(dim=-1) + 1e-3 * want.abs().max())
        assert rel.max().item() < 1e-2      # bf16 activations (2^-9 each) and rows of y (2^-9): 4e-3 at most of their norms' quotient


def test_a_limit_belongs_to_a_gate(pkg, device):
    mx, x, w = pkg.mixers, rand(4, 64).to(device), rand(32, 64).to(device)
    for act, limit in ((mx.ACT_NONE, 1.0), (mx.ACT_GELU, 1.0), (mx.ACT_SILU_GATE, -1.0), (mx.ACT_SILU_GATE, float("nan"))):
        with pytest.raises(RuntimeError):
            mx.few_rows(x, w, act, always=True, limit=limit)
    a = pkg.capi.LinearArgs(rows=1, K=8, N=8, groups=1, act=pkg.capi.ACT_NONE)
    assert pkg.capi.load().l3ci_linear_gated(C.byref(a), 1.0, 0.0) == pkg.capi.ERR_INVALID


def test_where_places_are_taken(pkg):
    pay = pkg.mixers.moe_places_pay
    assert pay(8, 4, 4) and pay(1, 4, 4) and pay(32, 16, 4) and pay(24, 32, 4)
    assert not pay(33, 4, 4) and not pay(1, 16, 4) and not pay(12, 32, 4)
