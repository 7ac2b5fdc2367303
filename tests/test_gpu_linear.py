"""`l3ci_linear`: products of few rows with a weight matrix, against fp64 sums of the same bf16 inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _want(x, w, act, capi):
    y = x.double() @ w.double().T
    if act == capi.ACT_GELU:
        return 0.5 * y * (1.0 + torch.erf(y * 0.5 ** 0.5))
    if act == capi.ACT_TANH:
        return torch.tanh(y)
    if act == capi.ACT_SILU_GATE:
        n = w.shape[0] // 2
        return y[..., :n] * torch.sigmoid(y[..., :n]) * y[..., n:]
    return y


def _check(got, want, K, f32):
    """fp32 sums of K products of size about 1 / sqrt(K): the error of a sum is below sqrt(K) roundings of a partial sum of
    size about 1, and the activations' slopes are below 2; a bf16 result adds half of a unit in the last place, 2^-9."""
    err = (got.double() - want).abs()
    bound = 2.0 * K ** 0.5 * 2.0 ** -23 * (1.0 + want.abs()) + (0.0 if f32 else 2.0 ** -8) * want.abs() + 1e-6
    assert bool((err <= bound).all()), f"largest excess {(err - bound).max().item():.3g}"


# rows: the edges of the 8-, 16-, 32- and 64-column forms; K: one 8-column vector, ends inside a stage, more stages than the ring
# has; N: inside a tile, whole tiles and one row behind them, more tiles than CTAs
@pytest.mark.parametrize("split", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("rows,K,N", [(1, 8, 1), (1, 2048, 4), (2, 72, 128), (8, 2048, 300), (9, 136, 129), (16, 1000, 129), (17, 2048, 300), (32, 4096, 64), (33, 520, 1025),
                                      (64, 2048, 2048), (7, 136, 40000)])
@pytest.mark.parametrize("act", [0, 1, 2, 3])
def test_products_of_few_rows(capi, device, rows, K, N, act, split):
    g = torch.Generator(device=device).manual_seed(rows * 7919 + K + N)
    x = torch.randn(rows, K, generator=g, device=device).bfloat16()
    w = (torch.randn((2 if act == capi.ACT_SILU_GATE else 1) * N, K, generator=g, device=device) * K ** -0.5).bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device=device)
    for out_dtype in (torch.bfloat16, torch.float32):
        got = capi.linear(x, w, act, out_dtype=out_dtype, split=split, status=status)
        assert got.dtype == out_dtype and got.shape == (rows, N)
        _check(got, _want(x, w, act, capi), K, out_dtype == torch.float32)
    assert status.item() == 0


def test_rows_with_a_stride_and_what_does_not_apply(capi, device):
    g = torch.Generator(device=device).manual_seed(5)
    w = (torch.randn(96, 64, generator=g, device=device) / 8).bfloat16()
    big = torch.randn(5, 3, 160, generator=g, device=device).bfloat16()
    for x in (big[:, -1, 8:72], big[:, :, 16:80], big[:1, :, :64], big[:, :1, 96:]):
        _check(capi.linear(x, w), _want(x, w, 0, capi), 64, False)
    for x in (big[:, :2, :64], big[:, :, 4:68], big.float()[..., :64], big[..., :60], big.transpose(0, 1)[..., :64], big[:0, :, :64],
              torch.zeros(65, 64, dtype=torch.bfloat16, device=device)):
        weight = w if x.shape[-1] == 64 else w[:, :60]
        assert capi.linear(x, weight) is None
    assert capi.linear(big[..., :64], w[:, ::2]) is None and capi.linear(big[..., :64], w.float()) is None


@pytest.mark.parametrize("split", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("rows", [1, 8, 9, 16, 17, 33, 64])
def test_chain_of_products_under_programmatic_launch(capi, device, rows, gated, split):
    """Each product reads what the one before wrote, while its own weights were asked for ahead of it: the bits of plain launches,
    and within the bound of the sums of fp64."""
    g = torch.Generator(device=device).manual_seed(11)
    sizes = [(2048, 2048), (3072, 2048), (2048, 3072), (520, 2048), (2048, 520)] * 2
    act, n = (capi.ACT_SILU_GATE, 2) if gated else (capi.ACT_NONE, 1)
    ws = [(torch.randn(n * N, K, generator=g, device=device) * K ** -0.5).bfloat16() for N, K in sizes]
    x0 = torch.randn(rows, 2048, generator=g, device=device).bfloat16()

    def chain():
        xs = [x0]
        for w in ws:
            xs.append(capi.linear(xs[-1], w, act, split=split, early=True))
        return xs

    status = torch.zeros(1, dtype=torch.int32, device=device)
    torch.cuda.synchronize()                         # the weights are complete: they may be read ahead of the stream
    with capi.programmatic_launch(False):
        want = chain()
    torch.cuda.synchronize()
    for x, w in zip(want, ws):
        _check(capi.linear(x, w, act, split=split, status=status), _want(x, w, act, capi), x.shape[1], False)
    assert status.item() == 0
    with capi.programmatic_launch(True):
        for _ in range(5):
            for a, b in zip(chain(), want):
                assert torch.equal(a, b)


@pytest.mark.parametrize("rows,groups,K,N", [(1, 4, 256, 256), (8, 16, 128, 512), (33, 3, 72, 130), (64, 16, 512, 128)])
def test_groups_of_products(capi, device, rows, groups, K, N):
    g = torch.Generator(device=device).manual_seed(rows + groups)
    w = (torch.randn(groups, N, K, generator=g, device=device) * K ** -0.5).bfloat16()
    x = torch.randn(rows, groups, K + 8, generator=g, device=device).bfloat16()[..., :K].transpose(0, 1)
    want = torch.einsum("grk,gnk->grn", x.double(), w.double())
    _check(capi.linear(x, w), want, K, False)
    out = torch.empty(rows, groups, N, dtype=torch.bfloat16, device=device).transpose(0, 1)
    assert capi.linear(x.contiguous(), w, out=out) is out
    _check(out, want, K, False)


def _ext_want(x, w, gated):
    y = x.double() @ w.double().T
    n = w.shape[0] // 2
    return y[..., :n] * torch.sigmoid(y[..., :n]) * y[..., n:] if gated else y


@pytest.mark.parametrize("gated", [False, True])
def test_extension_takes_any_layout_of_its_input(ext, device, gated):
    """Broadcast, strided and ragged inputs: what one row stride describes goes to the kernel, the rest to torch's product."""
    g = torch.Generator(device=device).manual_seed(3)
    K = 64
    w = (torch.randn(96, K, generator=g, device=device) / 8).bfloat16()
    base = torch.randn(2, K, generator=g, device=device).bfloat16()
    big = torch.randn(5, 3, 160, generator=g, device=device).bfloat16()
    many = torch.randn(70, K, generator=g, device=device).bfloat16()
    for x in (base[:, None].expand(2, 3, K), base[None].expand(3, 2, K), base[:1].expand(5, K), base[:, None, None].expand(2, 2, 3, K), base[0],
              big[:, -1, 8:72], big[:, :, 16:80], big[:, :2, :K], big[:, :, 4:68], big.transpose(0, 1)[..., :K], big[:1, :, :K], many, many[:65],
              many[:64], base.t().contiguous().t(), many.as_strided((4, K), (8, 1))):
        got = ext.linear(x, w, gated=gated)
        want = _ext_want(x, w, gated)
        assert got.shape == want.shape
        # as in _check; above 64 rows the gate and the up row are rounded to bf16 before their product, and so is silu(gate): 3 x 2^-8
        assert bool(((got.double() - want).abs() <= 2.0 ** -6 * want.abs() + 2.0 ** -9).all())


def _burst(ext, device, make):
    """Products with weights that the kernel right in front writes, against the same products with the device idle between the two."""
    g = torch.Generator(device=device).manual_seed(8)
    x = torch.randn(8, 2048, generator=g, device=device).bfloat16()
    ins = [torch.randn(2, 4096, 2048, generator=g, device=device).bfloat16() for _ in range(4)]
    want = []
    for a in ins:
        w = make(a)
        torch.cuda.synchronize()
        want.append(ext.linear(x, w))
        torch.cuda.synchronize()
    for _ in range(5):
        got = [ext.linear(x, make(a)) for a in ins]
        for a, b in zip(got, want):
            assert torch.equal(a, b)


def test_weights_written_by_the_kernel_in_front(ext, device):
    """`early` is off unless asked for: the weights may be the result of the launch before."""
    ones = torch.ones(2048, dtype=torch.bfloat16, device=device)
    _burst(ext, device, lambda a: ext.silu_mul(a[0], a[1]))
    _burst(ext, device, lambda a: ext.rms_norm(a[0], ones, 1e-5))
    _burst(ext, device, lambda a: ext.linear(a[0][:64], a[1][:2048]))
    _burst(ext, device, lambda a: a[0].clone().mul_(0.5))


def test_results_of_other_types_and_layouts_are_refused(capi, device):
    g = torch.Generator(device=device).manual_seed(4)
    x, w = torch.randn(4, 64, generator=g, device=device).bfloat16(), (torch.randn(24, 64, generator=g, device=device) / 8).bfloat16()

    def empty(*shape, dtype=torch.bfloat16, dev=device):
        return torch.empty(*shape, dtype=dtype, device=dev)

    with pytest.raises(ValueError):
        capi.linear(x, w, out_dtype=torch.float16)
    for out in (empty(4, 24, dtype=torch.float16), empty(4, 16), empty(5, 24), empty(4, 24, dev="cpu"), empty(4, 48)[:, ::2], empty(24, 4).t(),
                empty(1, 24).expand(4, 24), empty(2, 2, 24)):
        with pytest.raises(ValueError):
            capi.linear(x, w, out=out)
    for out in (empty(4, 24), empty(4, 24, dtype=torch.float32), empty(4, 40)[:, 3:27], empty(8, 24)[::2]):
        assert capi.linear(x, w, out=out) is out
        _check(out, _want(x, w, 0, capi), 64, out.dtype == torch.float32)
    # one x for all groups: not the kernel's
    assert capi.linear(x[None].expand(3, 4, 64), w[None].expand(3, 24, 64).contiguous()) is None


def test_a_wait_that_runs_out_has_a_place_to_be_reported(capi, ext, device):
    """Calls with and without a status word of their own leave both at zero (no wait of theirs can be made to run out: that would
    need a copy that never lands)."""
    g = torch.Generator(device=device).manual_seed(6)
    x, w = torch.randn(9, 2048, generator=g, device=device).bfloat16(), torch.randn(256, 2048, generator=g, device=device).bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device=device)
    capi.linear(x, w, status=status)
    ext.linear(x, w)
    assert ext.linear_status(x) == 0 and capi.load().l3ci_linear_poll(None) == capi.OK and status.item() == 0


@pytest.mark.parametrize("rows", [0, 1, 64, 65, 130])
@pytest.mark.parametrize("N", [0, 1, 12, 16])
def test_gated_products_of_any_width_and_number_of_rows(ext, device, rows, N):
    g = torch.Generator(device=device).manual_seed(rows + N)
    x, w = torch.randn(rows, 64, generator=g, device=device).bfloat16(), (torch.randn(2 * N, 64, generator=g, device=device) / 8).bfloat16()
    got, want = ext.linear(x, w, gated=True), _ext_want(x, w, True)
    assert got.shape == (rows, N) and bool(((got.double() - want).abs() <= 2.0 ** -6 * want.abs() + 2.0 ** -9).all())   # as above


def test_where_the_kernel_for_few_rows_is_taken(ext, capi, device):
    """The lines of the rule: rows against K, few and very many outputs, weights that are not read early; a fused activation always."""
    def taken(rows, N, K, act=0, early=True, groups=0):
        x = torch.zeros(*((groups,) if groups else ()), rows, K, dtype=torch.bfloat16, device=device)
        w = torch.zeros(*((groups,) if groups else ()), 2 * N if act == capi.ACT_SILU_GATE else N, K, dtype=torch.bfloat16, device=device)
        return ext.few_rows(x, w, act, early) is not None

    for rows, N, K, act, early, groups, want in (
            (16, 2048, 128, 0, True, 0, True), (17, 2048, 128, 0, True, 0, False), (8, 2048, 128, 0, False, 0, True), (9, 2048, 128, 0, False, 0, False),
            (32, 2048, 2048, 0, True, 0, True), (33, 2048, 2048, 0, True, 0, False), (16, 2048, 2048, 0, False, 0, True), (17, 2048, 2048, 0, False, 0, False),
            (64, 2048, 4096, 0, True, 0, True), (64, 512, 128, 1, True, 0, True), (64, 512, 128, 2, False, 0, True), (64, 512, 128, 3, True, 0, True),
            (64, 256, 128, 0, True, 0, True), (64, 257, 128, 0, True, 0, False),
            (64, 128, 128, 0, True, 2, True), (64, 128, 128, 0, True, 3, False), (64, 32768, 8, 0, True, 0, True), (64, 32767, 8, 0, True, 0, False),
            (65, 128, 2048, 0, True, 0, False)):
        assert taken(rows, N, K, act, early, groups) == want, (rows, N, K, act, early, groups)
    x, w = torch.randn(64, 128, device=device).bfloat16(), torch.randn(512, 128, device=device).bfloat16()
    assert ext.few_rows(x, w) is None                       # a pass that waits for the host takes it all the same
    _check(ext.few_rows(x, w, always=True), _want(x, w, 0, capi), 128, False)
    assert ext.few_rows(torch.cat([x, x[:1]]), w, always=True) is None
