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


@pytest.mark.parametrize("rows,E,top,bad", [(8, 4, 4, [2]), (32, 4, 4, [0, 1, 3]), (9, 40, 38, [0, 7, 33, 39]), (200, 4, 3, [1, 2])])
def test_router_logits_without_numbers(pkg, device, rows, E, top, bad):
    """A token whose logits run out of numbers has every expert once all the same: no expert more pairs than it has places, all places
    within the products' rows, and the other tokens' results untouched."""
    mx, width, ff = pkg.mixers, 64, 40
    h, z = rand(rows, width, seed=1).to(device), rand(rows, E, seed=2, scale=5).float().to(device)
    odd = torch.arange(rows, device=device) % 3 == 1
    w, down = rand(E, 2 * ff, width, seed=3, scale=0.1).to(device), rand(E, width, ff, seed=4, scale=0.1).to(device)

    def run(z):
        experts, ranks, weights, counts = mx.moe_route(z, torch.zeros(E, device=device), top)
        assert bool((experts.sort(dim=1).values.diff(dim=1) > 0).all()) and int(experts.min()) >= 0 and int(experts.max()) < E
        assert int(counts.sum()) == rows * top and int(counts.max()) <= rows and int(ranks.max()) < rows and int(ranks.min()) >= 0
        if rows > 32:
            return experts, None
        x, part_rows = mx.moe_places(h, experts, ranks, E)
        assert part_rows.unique().numel() == rows * top and int(part_rows.max()) < rows * E
        y = mx.few_rows(mx.few_rows(x, w, mx.ACT_SILU_GATE, always=True, limit=0.7, alpha=1.702), down, always=True)
        stream = torch.zeros(rows, width, device=device)
        mx.residual_norm(y, stream, dtype=torch.bfloat16, part_rows=part_rows, part_weights=weights)
        return experts, stream

    without = torch.where(odd[:, None], torch.full_like(z, float("nan")).index_fill(1, torch.tensor([e for e in range(E) if e not in bad], device=device), 1.0), z)
    (experts, stream), (_, want) = run(without), run(z)
    assert bool((experts[odd][:, :E - len(bad)] == torch.tensor([e for e in range(E) if e not in bad], device=device)[:top]).all())
    if stream is not None:
        assert torch.equal(stream[~odd], want[~odd]) and bool(stream[odd].isnan().all()) and bool(want.isfinite().all())


def test_models_whose_products_are_others(pkg, device, monkeypatch):
    """A model in fp32 gathers once, by sorted rows."""
    from tests.rupotar_cases import case, weights
    c = case("mixed", smooth=True)
    model = pkg.rupotar.RupotarDecoder(None, pkg.rupotar.config_from_json(c), device, 1, 64, weights=weights(pkg, c, 3), dtype=torch.float32)
    monkeypatch.setattr(pkg.mixers, "moe_places", lambda *a: pytest.fail("places"))
    assert bool(model.extend("a", list(range(5)), range(5)).isfinite().all())


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
