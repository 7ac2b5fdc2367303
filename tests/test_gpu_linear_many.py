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
