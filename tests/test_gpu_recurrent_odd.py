"""The recurrences by chunks where their results could leave those of the scan token by token: numbers that are not finite, the call that chooses
chunks by itself on strided parts of wider rows, and how near both are to 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


def inputs(kind, device, B, T, H, G, D, V, decay, seed=0):
    g = torch.Generator(device=device).manual_seed(seed)

    def rand(*shape, dtype=F32):
        return torch.randn(*shape, generator=g, device=device).to(dtype)

    x = {"state": rand(B, H, D, V) * 0.3, "gate": rand(B, T, H, V, dtype=BF16)}
    if kind == "delta":
        x["q"], x["k"] = (torch.nn.functional.normalize(rand(B, T, G, D), dim=-1) * s for s in (D ** -0.5, 1.0))
        x["v"], x["beta"], x["norm"] = rand(B, T, H, V, dtype=BF16), torch.sigmoid(rand(B, T, H)), torch.rand(V, generator=g, device=device) + 0.5
        x["g"] = torch.exp(-decay * torch.rand(B, T, H, D, generator=g, device=device))
    else:
        for n in "qkvg":
            x[n] = rand(B, T, H, D, dtype=BF16)
        x["bonus"], x["g_bias"], x["norm"] = rand(H, D), rand(H * D) * 0.3 + decay, torch.rand(H, D, generator=g, device=device) + 0.5
    return x


def scan(pkg, monkeypatch, x, how, positions=None):
    """Outputs and state; how: "tokens", "chunks" or "rule" (what the call takes by itself, which must be chunks)."""
    mx, state, taken = pkg.mixers, x["state"].clone(), []
    B, T, H, V = x["v"].shape
    positions = torch.full((B,), 3, dtype=torch.int32, device=state.device) if positions is None else positions
    args = [x[n] for n in "qkvg"] + [state, positions, x["norm"], x["gate"]]
    more = {n: x[n] for n in ("beta", "bonus", "g_bias") if n in x}
    scratch = torch.empty(1 << 24, dtype=torch.uint8, device=state.device) if how == "chunks" else None
    with monkeypatch.context() as m:
        lib = mx.load()
        by_chunks = lib.l3ci_recurrent_scan_chunks
        m.setattr(lib, "l3ci_recurrent_scan_chunks", lambda *a: taken.append(1) or by_chunks(*a))
        if how == "tokens":
            m.setattr(lib, "l3ci_recurrent_scan_scratch_bytes", lambda a: 0)
        out = mx.recurrent_scan(*args, act=mx.SIGMOID, eps=1e-5, scratch=scratch, **more)
    assert bool(taken) == (how != "tokens")
    return out.view(B, T, H, V), state


@pytest.mark.parametrize("value", ["nan", "inf", "-inf"])
@pytest.mark.parametrize("where", ["q", "k", "v", "g", "beta", "state"])
@pytest.mark.parametrize("kind,D,V", [("delta", 64, 72), ("delta", 128, 64), ("mix", 64, 64), ("mix", 128, 128)])
def test_numbers_that_are_not_finite(pkg, device, monkeypatch, kind, D, V, where, value):
    """In the middle of a chunk and of the prompt: finite where the scan token by token is, NaN where it is; tokens, heads, sequences and columns
    that they do not reach keep their values.  (An infinity, of which the terms of a sum are infinities of either sign token by token and one
    infinity by chunks, leaves the head's row not finite either way; what the norm makes of the others in the row then differs.)"""
    if kind == "mix" and where == "beta":
        pytest.skip("the delta rule's")
    B, T, H, G = 2, 53, 4, 2 if kind == "delta" else 4
    x = inputs(kind, device, B, T, H, G, D, V, 0.3 if kind == "delta" else -2.0)
    # the NaN of this hardware's arithmetic
    bits = {"nan": 0x7FFFFFFF, "inf": 0x7F800000, "-inf": 0x7F800000 - 2 ** 31}[value]
    number = torch.tensor(bits, dtype=torch.int32, device=device).view(F32)
    if x[where].dtype == BF16:
        number = torch.tensor(bits >> 16, dtype=torch.int16, device=device).view(BF16)
    x[where][(0, 1, 5, 7) if where == "state" else (0, 21, 1, 5)[:x[where].dim()]] = number
    (out, state), (want_out, want_state) = scan(pkg, monkeypatch, x, "chunks"), scan(pkg, monkeypatch, x, "tokens")
    assert torch.equal(state.isfinite(), want_state.isfinite())
    rows, want_rows = out.isfinite().all(-1), want_out.isfinite().all(-1)
    assert torch.equal(rows, want_rows)
    # (time mixing's decay is a finite function of an infinity)
    assert bool(state.isfinite().all() and rows.all()) == (kind == "mix" and where == "g" and value != "nan")
    if value == "nan":
        assert torch.equal(out.isnan(), want_out.isnan()) and torch.equal(state.isnan(), want_state.isnan())
        assert bool(out.isnan().any()) and bool(out[1].isfinite().all()) and (where == "state" or bool(out[0, :21].isfinite().all()))
    # two roundings of an output to bf16 each (2^-8 of the largest of its head), sums of at most 128 + 53 terms of a state in fp32
    near = want_out.double().abs().amax(-1, keepdim=True)
    assert bool(((out.double() - want_out.double()).abs() <= 2 ** -7 * near)[want_rows].all())
    near = torch.where(want_state.isfinite(), want_state.double(), 0.0).abs().amax((-2, -1), keepdim=True)
    assert bool(((state.double() - want_state.double()).abs() <= 1e-5 * near)[want_state.isfinite()].all())


@pytest.mark.parametrize("kind", ["delta", "mix"])
def test_the_call_that_chooses_chunks(pkg, device, monkeypatch, kind):
    """As the layers call it: parts of wider rows, the memory its own.  The bits are those of contiguous tensors, near those token by token."""
    B, T, H, D, V = (2, 133, 16, 128, 128) if kind == "delta" else (3, 241, 32, 64, 64)
    x = inputs(kind, device, B, T, H, H, D, V, 0.3 if kind == "delta" else -2.0)

    def part(t, before, behind):                           # [B, T, heads, n] as columns of [B, T, before + heads * n + behind]
        wide = torch.full((B, T, before + t[0, 0].numel() + behind), float("nan"), dtype=t.dtype, device=device)
        wide[..., before:before + t[0, 0].numel()] = t.flatten(2)
        return wide[..., before:before + t[0, 0].numel()].view(t.shape)

    parts = dict(x, g=part(x["g"], 16, 8), v=part(x["v"], 8, 0), gate=part(x["gate"], 24, 8))
    if kind == "delta":                                    # q and k as halves of one row
        both = torch.stack([x["q"], x["k"]], dim=2)
        parts["q"], parts["k"] = both[:, :, 0], both[:, :, 1]
    else:
        parts["q"], parts["k"] = part(x["q"], 8, 40), part(x["k"], 40, 8)
    assert not parts["q"].is_contiguous() and not parts["g"].is_contiguous()
    (out, state), (same_out, same_state) = scan(pkg, monkeypatch, parts, "rule"), scan(pkg, monkeypatch, x, "rule")
    assert torch.equal(out, same_out) and torch.equal(state, same_state)
    want_out, want_state = scan(pkg, monkeypatch, x, "tokens")
    assert pkg.mixers.scan_status(out) == 0                # neither form's waits ran out
    near = want_out.double().abs().amax(-1, keepdim=True)
    assert bool(((out.double() - want_out.double()).abs() <= 2 ** -7 * near).all())
    assert ((state - want_state).norm() / want_state.norm()).item() < 2e-6


def test_a_full_device(pkg, device, monkeypatch):
    """No memory for the chunks: the scan token by token."""
    x = inputs("delta", device, 2, 133, 16, 16, 128, 128, 0.3)
    want = scan(pkg, monkeypatch, x, "tokens")
    empty = torch.empty

    def full(*size, **kw):
        if kw.get("dtype") == torch.uint8:
            raise torch.OutOfMemoryError("full")
        return empty(*size, **kw)

    with monkeypatch.context() as m:
        m.setattr(torch, "empty", full)
        state = x["state"].clone()
        out = pkg.mixers.recurrent_scan(*[x[n] for n in "qkvg"], state, torch.full((2,), 3, dtype=torch.int32, device=device), x["norm"], x["gate"],
                                        act=pkg.mixers.SIGMOID, eps=1e-5, beta=x["beta"])
    assert torch.equal(out.view(want[0].shape), want[0]) and torch.equal(state, want[1])


def exact(kind, x):
    """State after all tokens in float64."""
    S, out = x["state"].double(), {n: t.double() for n, t in x.items()}
    for t in range(x["v"].shape[1]):
        k, v = out["k"][:, t], out["v"][:, t]
        if kind == "delta":
            S = out["g"][:, t, :, :, None] * S
            v = out["beta"][:, t, :, None] * (v - (k[:, :, None] @ S)[:, :, 0])
            S = S + k[..., None] * v[:, :, None]
        else:
            decay = torch.exp(-torch.exp(out["g"][:, t] + out["g_bias"].view(out["g"].shape[2:])))
            S = decay[..., None] * S + k[..., None] * v[:, :, None]
    return S


@pytest.mark.parametrize("kind,decay", [("delta", 0.0), ("delta", 1e-3), ("delta", 0.1), ("delta", 1.0), ("delta", 10.0), ("mix", -8.0), ("mix", -3.0),
                                        ("mix", -1.0), ("mix", 1.0)])
@pytest.mark.parametrize("T", [48, 1008])
@pytest.mark.parametrize("D", [64, 128])
def test_states_as_near_to_64_bits_as_token_by_token(pkg, device, monkeypatch, kind, decay, T, D):
    """Whatever the decay.  (The fp32 sums of both are in different orders: their errors' norms, over 4 x 2 heads' states, are within a tenth where the
    rounding of the last tokens is all there is; products on cut-off accumulators are twice as far off there.)"""
    x = inputs(kind, device, 2, T, 4, 4, D, D, decay, seed=T + D)
    want = exact(kind, x)
    chunks, tokens = ((scan(pkg, monkeypatch, x, how)[1].double() - want).norm().item() for how in ("chunks", "tokens"))
    assert chunks <= 1.1 * tokens, (chunks / want.norm().item(), tokens / want.norm().item())
