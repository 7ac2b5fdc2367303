"""Products of many rows with their activation over pairs of SMs (`l3ci_linear_many`): edges of the 256 x 256 tiles and of the 64-column
stages, strides, every activation, against the fp32 product of the same bf16 operands."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def rand(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16().cuda()


def many(capi, x, w, act, out):
    N = w.shape[0] // (2 if act == capi.ACT_SILU_GATE else 1)
    a = capi.LinearArgs(x=x.data_ptr(), w=w.data_ptr(), out=out.data_ptr(), rows=x.shape[0], x_st=x.stride(0), out_st=out.stride(0), K=w.shape[1], N=N,
                        groups=1, act=act, stream=torch.cuda.current_stream().cuda_stream)
    return capi.load().l3ci_linear_many(C.byref(a))


def want_of(capi, x, w, act):
    y = x.float() @ w.float().T
    if act == capi.ACT_SILU_GATE:
        g, u = y.chunk(2, dim=-1)
        return g / (1 + torch.exp(-g)) * u
    return torch.nn.functional.gelu(y) if act == capi.ACT_GELU else torch.tanh(y) if act == capi.ACT_TANH else y


@pytest.mark.parametrize("act", [0, 1, 2, 3])
@pytest.mark.parametrize("rows,K,N", [(1, 64, 8), (127, 72, 136), (128, 8, 128), (129, 320, 256), (255, 2048, 264), (256, 384, 512), (257, 640, 1032),
                                      (600, 1000, 2056), (3000, 512, 4096)])
def test_products_with_activations(capi, device, rows, K, N, act):
    torch.backends.cuda.matmul.allow_tf32 = False
    gated = act == capi.ACT_SILU_GATE
    wide, w = rand(rows, K + 24, seed=1), rand((2 if gated else 1) * N, K, seed=2, scale=2 * K ** -0.5)
    x = wide[:, 8:8 + K]
    out = torch.full((rows, N + 8), 7.0, dtype=BF16, device=device)
    assert many(capi, x, w, act, out[:, :N]) == capi.OK
    want = want_of(capi, x, w, act)
    err = (out[:, :N].double() - want.double()).norm(dim=-1) / (want.double().norm(dim=-1) + 1e-3 * want.abs().max())
    assert err.max().item() < 6e-3                      # one rounding to bf16: 2^-9 of a value, rows of few values included
    assert bool((out[:, N:] == 7.0).all())
    first = out.clone()
    assert many(capi, x, w, act, out[:, :N]) == capi.OK and torch.equal(first, out)
    assert capi.load().l3ci_linear_poll(torch.cuda.current_stream().cuda_stream) == capi.OK


@pytest.mark.parametrize("rows,K,N", [(300, 640, 1032), (2049, 2048, 8192)])
def test_silu_mul_of_a_product_bit_for_bit(ext, capi, device, rows, K, N):
    """The form that stands for a bf16 product and silu_mul: their bits, where this kernel's sums are the plain product's."""
    x, w = rand(rows, K, seed=3), rand(2 * N, K, seed=4, scale=8 * K ** -0.5)
    plain, out = torch.empty(rows, 2 * N, dtype=BF16, device=device), torch.empty(rows, N, dtype=BF16, device=device)
    a = capi.LinearArgs(x=x.data_ptr(), w=w.data_ptr(), out=out.data_ptr(), rows=rows, x_st=K, out_st=N, K=K, N=N, groups=1, act=4,
                        stream=torch.cuda.current_stream().cuda_stream)
    assert many(capi, x, w, 0, plain) == capi.OK and capi.load().l3ci_linear_many(C.byref(a)) == capi.OK
    assert torch.equal(out, ext.silu_mul(plain[:, :N], plain[:, N:]))


def test_refused(capi, device):
    x, w, out = rand(300, 64), rand(64, 64), torch.empty(300, 64, dtype=BF16, device=device)
    assert many(capi, x[:, :60], w[:, :60], 0, out) == capi.ERR_ALIGNMENT
    assert many(capi, x, w, 5, out) == capi.ERR_INVALID
    assert many(capi, x[:1].expand(300, 64), w, 0, out) == capi.ERR_INVALID
    assert many(capi, x, w[:60], 0, out[:, :60]) == capi.ERR_ALIGNMENT


def every_number(device):
    """The finite bf16 numbers, 255 x 256."""
    bits = torch.arange(65536, dtype=torch.int32)
    return bits[(bits & 0x7F80) != 0x7F80].to(torch.int16).view(BF16).view(255, 256).to(device)


def sums(x, up=None):
    """Operands whose product's sums are x, one term each (and, gated, `up`)."""
    eye = torch.eye(256, dtype=BF16, device=x.device)
    if up is None:
        return x, eye
    one = torch.zeros(x.shape[0], 8, dtype=BF16, device=x.device)
    one[:, 0] = up
    pick = torch.zeros(256, 264, dtype=BF16, device=x.device)
    pick[:, 256] = 1.0
    return torch.cat([x, one], 1), torch.cat([torch.cat([eye, torch.zeros(256, 8, dtype=BF16, device=x.device)], 1), pick])


@pytest.mark.parametrize("act", [1, 2, 3])
def test_activation_of_every_number(capi, device, act):
    """One rounding to bf16 (2^-8 of a value) and at most 1e-5 of it, tails included; numbers below the least normal may be zeros, and silu is
    zero where exp(-z) is no fp32 number."""
    x = every_number(device)
    a, w = sums(x, 1.0 if act == capi.ACT_SILU_GATE else None)
    out, z = torch.empty(255, 256, dtype=BF16, device=device), x.double()
    assert many(capi, a, w, act, out) == capi.OK
    want = 0.5 * z * torch.special.erfc(-z * 0.5 ** 0.5) if act == capi.ACT_GELU else torch.tanh(z) if act == capi.ACT_TANH else z * torch.sigmoid(z)
    bound = (2 ** -8 + 1e-5) * want.abs() + (3e-37 if act == capi.ACT_SILU_GATE else 2e-38)
    assert bool(((out.double() - want).abs() <= bound).all())


def test_gate_of_sums_as_in_few_rows(capi, device):
    """silu(z) u with the bits of the product of few rows, which has expf and the full division: every bf16 number, and z of 24 bits where exp(-z) is
    large, whose rounding a shorter exponential moves now and then."""
    g = torch.Generator(device=device).manual_seed(5)
    z = torch.cat([every_number(device).float(), -85 * torch.rand(4097, 256, generator=g, device=device)])
    first = z.bfloat16()
    a, w = sums(first, -1.375)
    second = torch.where(z.abs() < 100, z - first.float(), 0.0).bfloat16()
    a, w = torch.cat([a, second], 1), torch.cat([w, torch.cat([torch.eye(256), torch.zeros(256, 256)]).to(device, BF16)], 1)
    out, few = torch.empty_like(first), torch.empty_like(first)
    assert many(capi, a, w, capi.ACT_SILU_GATE, out) == capi.OK
    for r in range(0, a.shape[0], 64):
        part, to = a[r:r + 64], few[r:r + 64]
        args = capi.LinearArgs(x=part.data_ptr(), w=w.data_ptr(), out=to.data_ptr(), rows=part.shape[0], x_st=520, out_st=256, K=520, N=256, groups=1,
                               act=capi.ACT_SILU_GATE, stream=torch.cuda.current_stream().cuda_stream)
        assert capi.load().l3ci_linear(C.byref(args)) == capi.OK
    assert torch.equal(out.view(torch.int16), few.view(torch.int16))


def test_silu_mul_of_every_number(ext, capi, device):
    x = every_number(device) + 0.0                      # (a sum is never -0)
    a, w = sums(x, 1.375)
    out, up = torch.empty(255, 256, dtype=BF16, device=device), torch.full_like(x, 1.375)
    args = capi.LinearArgs(x=a.data_ptr(), w=w.data_ptr(), out=out.data_ptr(), rows=255, x_st=264, out_st=256, K=264, N=256, groups=1, act=4,
                           stream=torch.cuda.current_stream().cuda_stream)
    assert capi.load().l3ci_linear_many(C.byref(args)) == capi.OK
    assert torch.equal(out.view(torch.int16), ext.silu_mul(x, up).view(torch.int16))


@pytest.mark.parametrize("act", [1, 2, 3, 4])
def test_sums_that_are_not_finite(ext, pkg, capi, device, act):
    """NaN where the activation of its own on a bf16 product has it."""
    mx, odd = pkg.mixers, [float("nan"), float("inf"), -float("inf")]
    w = torch.cat([torch.eye(256, dtype=BF16, device=device)] * (2 if act > 2 else 1))
    x = torch.zeros(300, 256, dtype=BF16, device=device)
    for r in range(300):
        x[r, r % 256] = odd[r % 3]
    out, plain = torch.empty(300, 256, dtype=BF16, device=device), torch.empty(300, w.shape[0], dtype=BF16, device=device)
    args = capi.LinearArgs(x=x.data_ptr(), w=w.data_ptr(), out=out.data_ptr(), rows=300, x_st=256, out_st=256, K=256, N=256, groups=1, act=act,
                           stream=torch.cuda.current_stream().cuda_stream)
    assert capi.load().l3ci_linear_many(C.byref(args)) == capi.OK and many(capi, x, w, 0, plain) == capi.OK
    want = (mx.gelu_(plain) if act == 1 else mx.tanh_(plain) if act == 2 else mx.gated_act(plain) if act == 3 else
            ext.silu_mul(plain[:, :256], plain[:, 256:]))
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out[~out.isnan()], want[~want.isnan()])


@pytest.mark.parametrize("B,T", [(1, 2048), (2, 1000)])
def test_the_calls_that_choose_it(ext, capi, device, B, T):
    """`many_rows` and a gated `linear` on a part of wider rows: the bits of the C call, near the fp32 product."""
    K, N = 512, 2048
    wide, w = rand(B, T, K + 64, seed=7), rand(2 * N, K, seed=8, scale=2 * K ** -0.5)
    x = wide[..., 32:32 + K]
    y = x.reshape(B * T, K)
    for act, rows, got in ((capi.ACT_GELU, w, ext.many_rows(x, w, capi.ACT_GELU)), (capi.ACT_SILU_GATE, w, ext.many_rows(x, w, capi.ACT_SILU_GATE)),
                           (4, w, ext.linear(x, w, gated=True))):
        n = N if act > 2 else 2 * N
        assert got is not None and got.shape == (B, T, n)
        out = torch.empty(B * T, n, dtype=BF16, device=device)
        args = capi.LinearArgs(x=y.data_ptr(), w=rows.data_ptr(), out=out.data_ptr(), rows=B * T, x_st=y.stride(0), out_st=n, K=K, N=n, groups=1, act=act,
                               stream=torch.cuda.current_stream().cuda_stream)
        assert capi.load().l3ci_linear_many(C.byref(args)) == capi.OK and torch.equal(got.view(B * T, n), out)
        want = want_of(capi, y, rows, capi.ACT_SILU_GATE if act == 4 else act).double()
        assert ((out.double() - want).norm() / want.norm()).item() < 6e-3
