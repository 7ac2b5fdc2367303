"""The recurrences by chunks of 16 tokens (`l3ci_recurrent_scan_chunks`) against the float64 restatement: chunks and segments that end early, column
blocks that are not full, shared key heads, carried and fresh states, decays that leave nothing and those that keep everything."""
import ctypes as C

import pytest
import torch

from oracle import rupotar as ref

pytestmark = pytest.mark.gpu
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


def rand(*shape, seed=0, scale=1.0, dtype=BF16):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


def close(got, want, bound, what):
    rel = (got.double().cpu() - want).norm(dim=-1) / (want.norm(dim=-1) + 1e-3 * want.abs().max() + 1e-30)
    assert torch.isfinite(got.double()).all() and rel.max().item() < bound, (what, rel.max().item())


def memory(chunks, bytes_of_one, device):
    return torch.full((chunks * bytes_of_one + 8,), 255, dtype=torch.uint8, device=device)[:chunks * bytes_of_one]     # (what it holds before is NaN)


# bytes of a chunk of one head: 16 rows of D floats each of Q and K (the delta rule's W), 16 of 16 of M (T), D decays
def one(heads, D, delta):
    return 4 * heads * ((3 if delta else 2) * 16 * D + (2 if delta else 1) * 256 + D)


@pytest.mark.parametrize("chunks", [1, 2, 100])
@pytest.mark.parametrize("T", [1, 15, 16, 17, 50])
@pytest.mark.parametrize("H,G,D,V,decay", [(4, 2, 64, 96, 1.0), (2, 2, 128, 128, 1.0), (3, 1, 128, 8, 40.0), (2, 1, 64, 192, 0.0)])
def test_delta_rule(pkg, device, H, G, D, V, decay, T, chunks):
    B, eps = 2, 1e-4
    q, k = (torch.nn.functional.normalize(rand(B, T, G, D, seed=s, dtype=F32), dim=-1) for s in (1, 2))
    v, gate, norm = rand(B, T, H, V, seed=3), rand(B, T, H, V, seed=4), rand(V, seed=5, dtype=F32)
    g = torch.exp(-decay * torch.rand(B, T, H, D, generator=torch.Generator().manual_seed(6)))
    beta, held = torch.sigmoid(rand(B, T, H, seed=7, dtype=F32)), rand(B, H, D, V, seed=8, dtype=F32)
    pos = torch.tensor([0, 9], dtype=torch.int32)
    state, status = held.to(device), torch.zeros(1, dtype=torch.int32, device=device)
    tail, conv = torch.full((B, 2, 2 * G * D + H * V), 7.0, dtype=BF16, device=device), rand(B, T, 2 * G * D + H * V, seed=9).to(device)
    before = tail.clone()
    d = [t.to(device) for t in (q, k, v, g, norm, gate, beta, pos)]
    out = pkg.mixers.recurrent_scan(*d[:4], state, d[7], d[4], d[5], act=pkg.mixers.SIGMOID, eps=eps, beta=d[6], conv_in=conv, tail=tail, taps=3, status=status,
                                    scratch=memory(chunks, one(B * H, D, True), device))
    assert status.item() == 0
    of = [i // (H // G) for i in range(H)]
    for b in range(B):
        start = torch.zeros(H, D, V, dtype=F64) if b == 0 else held[b].double()
        o, S = ref.delta_scan(*(t[b].double() for t in (q[:, :, of], k[:, :, of], v, g, beta)), state=start)
        want = ref.rms(o, eps) * norm.double() / (1 + torch.exp(-gate[b].double()))
        # heads whose output nearly cancels blow the sums' rounding up: against the head's values, not the normed output
        scale = ref.rms(o, eps).abs().max()
        assert (out[b].view(T, H, V).double().cpu() - want).abs().max() < 1e-2 * scale * norm.abs().max(), (b, "out")
        close(state[b].reshape(1, -1), S.reshape(1, -1), 2e-6, (b, "state"))
        if T >= 2:
            assert torch.equal(tail[b], conv[b, T - 2:])
        else:
            assert torch.equal(tail[b, 1], conv[b, 0]) and bool((tail[b, 0] == (0.0 if b == 0 else before[b, 1])).all())


@pytest.mark.parametrize("chunks", [1, 3, 100])
@pytest.mark.parametrize("T", [1, 16, 31, 70])
@pytest.mark.parametrize("H,D,bias", [(4, 64, -2.0), (2, 128, -2.0), (3, 64, 3.0), (2, 64, -20.0)])
def test_time_mixing(pkg, device, H, D, bias, T, chunks):
    B, eps = 2, 1e-4
    r, k, v, gate, x = (rand(B, T, H, D, seed=s) for s in range(5))
    w0, u, norm, held = rand(H * D, seed=6, dtype=F32) + bias, rand(H, D, seed=7, dtype=F32), rand(H, D, seed=8, dtype=F32), rand(B, H, D, D, seed=9, dtype=F32)
    state, status = held.to(device), torch.zeros(1, dtype=torch.int32, device=device)
    d = [t.to(device) for t in (r, k, v, x, norm, gate, u, w0)]
    out = pkg.mixers.recurrent_scan(*d[:4], state, torch.tensor([3, 0], dtype=torch.int32, device=device), d[4], d[5], act=pkg.mixers.SILU, eps=eps, bonus=d[6],
                                    g_bias=d[7], status=status, scratch=memory(chunks, one(B * H, D, False), device))
    assert status.item() == 0
    for b in range(B):
        S = torch.zeros(H, D, D, dtype=F64) if b == 1 else held[b].double()
        w = torch.exp(-torch.exp(x[b].double() + w0.double().view(H, D)))
        want = torch.empty(T, H, D, dtype=F64)
        for t in range(T):
            kv = k[b, t].double()[:, :, None] * v[b, t].double()[:, None]
            want[t] = (r[b, t].double()[:, None] @ (S + u.double()[:, :, None] * kv))[:, 0]
            S = w[t][:, :, None] * S + kv
        want = ref.rms(want, eps) * norm.double() * ref.silu(gate[b].double())
        close(out[b].view(T, H, D), want, 2e-2, (b, "out"))
        close(state[b].reshape(1, -1), S.reshape(1, -1), 2e-6, (b, "state"))


def test_where_chunks_are_taken(pkg, device):
    lib, A = pkg.mixers.load(), pkg.mixers.RecurrentScanArgs

    def need(B, T, H, D, V, kind=0, dtype=0, shift=0):
        a = A(**{n: 4096 + shift for n in "q k v g beta bonus g_bias norm gate state out positions".split()})
        a.B, a.T, a.H, a.G, a.D, a.V, a.kind, a.dtype = B, T, H, H, D, V, kind, dtype
        a.qk_st = a.v_st = a.g_st = a.gate_st = a.out_st = H * D
        a.qk_sh = a.v_sh = a.g_sh = a.gate_sh = a.out_sh = D
        a.state_sb = H * D * V
        return lib.l3ci_recurrent_scan_scratch_bytes(C.byref(a))

    assert need(2, 132, 16, 128, 128) == 9 * one(32, 128, True) and need(2, 131, 16, 128, 128) == 0 and need(1, 6000, 16, 128, 128) == 0
    assert need(3, 59, 16, 128, 128) == 4 * one(48, 128, True) and need(16, 39, 16, 128, 128) == 0
    assert need(3, 240, 32, 64, 64, kind=1) == 15 * one(96, 64, False) and need(3, 239, 32, 64, 64, kind=1) == need(2, 6000, 32, 64, 64, kind=1) == 0
    assert need(16, 79, 16, 128, 128) == 0 and need(16, 80, 16, 128, 128) == 5 * one(256, 128, True)
    assert 0 < need(8, 6000, 16, 128, 128) <= 256 << 20                             # longer prompts: segments
    assert need(3, 1000, 16, 128, 128, dtype=1) == need(3, 1000, 16, 32, 128) == need(3, 1000, 16, 128, 124) == need(3, 1000, 16, 128, 128, shift=2) == 0
    a = A()
    assert lib.l3ci_recurrent_scan_chunks(C.byref(a), None, 0) != 0
