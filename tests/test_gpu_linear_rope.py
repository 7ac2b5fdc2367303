"""The projections of a step with rotation and cache write (`linear_rot_embed_kv_cache`) against the product in fp32 and the rotation of its
sums, and bit for bit against the two calls that it stands for: rows of every form of the product, portions of several tokens, both
numbers of CTAs a tile, positions outside the table or the cache."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def rand(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16().cuda()


@pytest.mark.parametrize("B,T", [(1, 1), (3, 1), (8, 1), (9, 1), (2, 5), (17, 1), (32, 1)])
@pytest.mark.parametrize("Hq,Hkv,D,K", [(32, 8, 64, 2048), (16, 4, 128, 1024), (3, 1, 64, 1032), (64, 8, 64, 512)])
def test_projections_rotated(ext, device, B, T, Hq, Hkv, D, K):
    L, rows = 40, 50
    x, w = rand(B, T, K, seed=1), rand((Hq + 2 * Hkv) * D, K, seed=2, scale=K ** -0.5)
    freq = torch.randn(rows, D, generator=torch.Generator().manual_seed(3)).cuda()
    pos = torch.tensor([(7 * b) % (L - T) for b in range(B)], dtype=torch.int32, device=device)
    pos[-1] = L - 1 if T > 1 else L                    # its last tokens, or its only one, do not fit the cache
    ck, cv = (torch.full((B + 1, L, Hkv, D), 7.0, dtype=BF16, device=device) for _ in range(2))
    q = ext.linear_rot_embed_kv_cache(x, w, freq, ck, cv, Hq, Hkv, pos, early=True, always=True)
    assert q is not None and q.shape == (B, T, Hq, D)
    y = (x.float() @ w.float().T).view(B, T, Hq + 2 * Hkv, D)
    qf, kf, vf = y.split([Hq, Hkv, Hkv], dim=2)

    def turn(t, p):                                    # [heads, D] at position p
        c, s = freq[p, 0::2], freq[p, 1::2]
        a, b = t[..., 0::2], t[..., 1::2]
        return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)

    def close(got, want):
        assert ((got.float() - want).norm() / want.norm()).item() < 6e-3          # two roundings to bf16

    ck2, cv2 = (torch.full_like(c, 7.0) for c in (ck, cv))
    q2 = ext.rot_embed_kv_cache(ext.linear(x, w, early=True, always=True), freq, ck2, cv2, 0, Hq, Hkv, positions=pos)
    fits = torch.tensor([[int(pos[b]) + t < L for t in range(T)] for b in range(B)], device=device)
    assert torch.equal(q[fits], q2[fits]) and torch.equal(ck, ck2) and torch.equal(cv, cv2)
    for b in range(B):
        for t in range(T):
            p = int(pos[b]) + t
            if p >= L:
                continue
            close(q[b, t], turn(qf[b, t], p))
            close(ck[b, p], turn(kf[b, t], p))
            close(cv[b, p], vf[b, t])
            ck[b, p], cv[b, p] = 7.0, 7.0
    assert bool((ck == 7.0).all()) and bool((cv == 7.0).all())


def test_an_infinite_value_stays_in_its_place(ext, device):
    x, w, freq = torch.ones(1, 1, 2048, dtype=BF16, device=device), rand(48 * 64, 2048, scale=0.02), torch.randn(10, 64, device=device)
    w[-1], w[-4] = 1e38, -1e38                                 # sums beyond fp32
    pos = torch.zeros(1, dtype=torch.int32, device=device)
    a, b = ([torch.zeros(1, 8, 8, 64, dtype=BF16, device=device) for _ in range(2)] for _ in range(2))
    q = ext.linear_rot_embed_kv_cache(x, w, freq, *a, 32, 8, pos, always=True)
    q2 = ext.rot_embed_kv_cache(ext.linear(x, w, always=True), freq, *b, 0, 32, 8, positions=pos)
    assert torch.equal(q, q2) and torch.equal(a[0], b[0]) and torch.equal(a[1], b[1]) and a[1][0, 0, 7, -1].isinf() and a[1][0, 0, 7, -4].isinf()


def test_where_it_does_not_apply(ext, device):
    w, freq = rand(48 * 64, 2048), torch.zeros(10, 64, device=device)
    caches = [torch.zeros(64, 8, 8, 64, dtype=BF16, device=device) for _ in range(2)]

    def call(x, w=w, always=True):
        return ext.linear_rot_embed_kv_cache(x, w, freq, *caches, 32, 8, torch.zeros(x.shape[0], dtype=torch.int32, device=device), always=always)

    assert call(rand(33, 1, 2048)) is None                                         # more rows than the last step has threads for
    assert call(rand(32, 1, 2048), always=False) is None and call(rand(8, 1, 2048), always=False) is not None     # the rule of `linear`
    assert call(rand(1, 1, 256), w[:, :256].contiguous()) is None                  # too few stages for clusters
    assert call(rand(2, 1, 4096)[..., 1:2049]) is None                             # rows that do not start on 16 bytes
    with pytest.raises(RuntimeError):
        call(rand(1, 1, 1024))
