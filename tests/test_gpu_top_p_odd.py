"""Nucleus sampling of rows whose logits hold NaN, infinities or values whose scaled difference overflows: a step still takes one
token of the vocabulary per row and moves every counter by one, the same in every run, and leaves the other rows alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu
NAN, INF = float("nan"), float("inf")


def _rows(kind, rows, vocab, device):
    g = torch.Generator(device=device).manual_seed(rows + vocab)
    x = torch.randn(rows, vocab, generator=g, device=device) * 3
    some = torch.rand(rows, vocab, generator=g, device=device) < 0.02
    some[:, vocab // 3] = True
    odd = torch.ones(rows, dtype=torch.bool, device=device)
    odd[1::2] = False                                       # every other row is an ordinary one
    value = {"nan": NAN, "nan_all": NAN, "inf": INF, "inf_all": INF, "ninf_all": -INF, "huge": 3.3e38, "lowest_all": torch.finfo(torch.bfloat16).min}[kind]
    x = torch.where(odd[:, None] & (some | kind.endswith("_all")), value, x)
    return x.bfloat16(), odd


def _run(capi, x, calls=3):
    rows, dev = x.shape[0], x.device
    out, i64, i32 = torch.full((rows, calls + 2), -1, dtype=torch.int64, device=dev), dict(dtype=torch.int64, device=dev), dict(dtype=torch.int32, device=dev)
    steps, cur, pos, lens, count = (torch.zeros(rows, **d) for d in (i64, i64, i32, i32, i32))
    mass = torch.zeros(rows, device=dev)
    for _ in range(calls):
        capi.top_p_step(x, 0.8, 0.9, 5, out, steps, cur, pos, lens, count, mass)
    return out, steps, cur, pos, lens, count, mass


@pytest.mark.parametrize("rows,vocab", [(1, 37), (12, 5001), (30, 5001), (40, 37), (60, 70000), (80, 5001), (80, 70000), (9, 300000)])
@pytest.mark.parametrize("kind", ["nan", "nan_all", "inf", "inf_all", "ninf_all", "huge", "lowest_all"])
def test_one_token_per_row_and_step(capi, device, kind, rows, vocab):
    x, odd = _rows(kind, rows, vocab, device)
    first, again = _run(capi, x), _run(capi, x)
    out, steps, cur, pos, lens, count, mass = first
    for t in (steps, pos, lens):
        assert bool((t == 3).all())
    assert bool(((out[:, :3] >= 0) & (out[:, :3] < vocab)).all()) and bool((out[:, 3:] == -1).all()) and torch.equal(out[:, 2], cur)
    for a, b in zip(first, again):
        assert torch.equal(a.nan_to_num(-7.0), b.nan_to_num(-7.0))
    if kind in ("nan_all", "ninf_all", "inf_all"):          # no logit differs from another: the first one stands in
        assert bool((out[odd, :3] == 0).all())
    # the ordinary rows among them: what they give with ordinary neighbours
    y = torch.where(odd[:, None], torch.zeros_like(x), x)
    for a, b in zip(first, _run(capi, y)):
        assert torch.equal(a[~odd], b[~odd])


@pytest.mark.parametrize("pattern", [-1, -64])           # 0xFFFF, 0xFFC0: NaN with the sign set, in order below every number
@pytest.mark.parametrize("rows,vocab", [(1, 5001), (20, 70000), (40, 5001), (75, 70000)])
def test_a_negative_nan_in_one_share_of_the_row(capi, device, rows, vocab, pattern):
    """The boundary of the nucleus is then below all that the other shares hold: by counts as by masses (a tail of -inf, above the boundary
    too, takes the row there)."""
    long = 8 * 8191 * 8 + 8
    x = (torch.randn(rows, vocab, generator=torch.Generator(device=device).manual_seed(vocab), device=device) * 3).bfloat16()
    x.view(torch.int16)[torch.arange(rows, device=device), torch.arange(rows, device=device) * 997 % vocab] = pattern
    wide = torch.full((rows, long), -INF, dtype=torch.bfloat16, device=device)
    wide[:, :vocab] = x
    got, want = _run(capi, x), _run(capi, wide)
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a + (long - vocab if i == 5 else 0), b)
