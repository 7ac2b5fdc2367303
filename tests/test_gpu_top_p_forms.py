"""The nucleus-sampling step by key counts against the same step by masses, which takes rows too long for the counts: an appended
tail of -inf logits has no mass, so a row and the row with that tail must give the same token, nucleus size and mass."""
import pytest
import torch

pytestmark = pytest.mark.gpu
LONG = 8 * 8191 * 8 + 8      # one group more than eight CTAs count


@pytest.mark.parametrize("rows,vocab", [(1, 8), (2, 1001), (40, 8191), (15, 65537), (16, 65536), (33, 128256), (74, 128256), (75, 65528), (75, 65529)])
@pytest.mark.parametrize("kind", ["normal", "flat", "steps", "holes"])
def test_counts_and_masses_agree(capi, device, rows, vocab, kind):
    g = torch.Generator(device=device).manual_seed(rows + vocab)
    x = torch.randn(rows, vocab, generator=g, device=device) * 2.5
    if kind == "flat":
        x.fill_(-1.25)
    elif kind == "steps":
        x = x.round()                                  # many ties at the boundary, zeros of both signs among them
    elif kind == "holes":
        x[torch.rand(rows, vocab, generator=g, device=device) < 0.9] = float("-inf")
        x[:, vocab // 2] = 3.0
    x = x.bfloat16()
    long = torch.full((rows, LONG), float("-inf"), dtype=torch.bfloat16, device=device)
    long[:, :vocab] = x

    def run(logits):
        out, i64, i32 = torch.zeros(rows, 2, dtype=torch.int64, device=device), dict(dtype=torch.int64, device=device), dict(dtype=torch.int32, device=device)
        steps, cur, pos, lens, count = (torch.zeros(rows, **d) for d in (i64, i64, i32, i32, i32))
        mass = torch.zeros(rows, device=device)
        for _ in range(2):
            capi.top_p_step(logits, 0.8, 0.9, 77, out, steps, cur, pos, lens, count, mass)
        return out, steps, pos, lens, count, mass

    odd = torch.empty(rows, vocab + 3, dtype=torch.bfloat16, device=device)      # rows that do not start on 16 bytes
    odd[:, 3:] = x
    want = run(long)
    for logits in (x, odd[:, 3:]):
        for a, b in zip(run(logits), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("kind", ["normal", "flat", "steps", "holes"])
@pytest.mark.parametrize("rows,vocab", [(75, 1), (75, 4096), (75, 4097), (149, 4100)])
def test_short_rows_of_one_cta(capi, device, rows, vocab, kind):
    test_counts_and_masses_agree(capi, device, rows, vocab, kind)


def test_the_form_taken(capi, device):
    """CTAs per row, + 16 by counts.  A launch that fails for another reason than its place on the device is an error, not the other form."""
    if torch.cuda.get_device_properties(device).multi_processor_count != 148:
        pytest.skip("the bounds are those of 148 SMs")
    choice = capi.load().l3ci_top_p_kernel_choice
    for rows, vocab, want in ((1, 8, 24), (15, 128256, 24), (16, 128256, 20), (33, 8, 20), (34, 128256, 18), (74, 65528, 18), (75, 65528, 17),
                              (75, 65529, 18), (75, 4097, 17), (75, 4096, 1), (256, 300000, 24), (1, LONG, 8), (33, LONG, 4), (80, LONG, 1)):
        assert choice(rows, vocab) == want, (rows, vocab)
    assert choice(0, 8) == choice(1, 0) == -1
