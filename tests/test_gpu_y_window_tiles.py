"""Window attention in tiles of four queries (cd_window_attention_rows where what they read is worth it) against 64 bits: rows that
are no multiple of four, one to eight blocks a tile (eight: 145 tokens behind 700), head counts on both sides of what a thread mixes
(8, 16, 32), two query heads and more (and an odd number) a key head, kept tokens, earlier keys from the ring. Three cases go one
query at a time: few bytes (145 tokens, 60 tokens), or more shared memory than two blocks on an SM have (32 heads of 128).

fp32 storage: sums of at most `dim` and `window` fp32 products and CUDA's expf and log1pf, 2e-6 of the row's largest value; bf16
storage adds its rounding of the result, 2^-8 of the value."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, ring_k, ring_v, r1, r2, talk, window, keep, pos0, scale):
    B, S, H, _ = q.shape
    G = k.shape[2]
    first = max(0, pos0 - window - keep)
    old = [j for j in range(pos0) if j < keep or j >= first]
    slot = [j if j < keep else keep + (j - keep) % window for j in old]
    pos = torch.tensor(old + list(range(pos0, pos0 + S)), device=q.device)
    kk = torch.cat([ring_k[:, slot], k], 1).double().repeat_interleave(H // G, 2)
    vv = torch.cat([ring_v[:, slot], v], 1).double().repeat_interleave(H // G, 2)
    i = torch.arange(pos0, pos0 + S, device=q.device)
    d = i[:, None] - pos[None]
    # a ring slot holds the newest position of its class: what the window no longer reaches is not seen either
    seen = (d >= 0) & ((d < window) | (pos[None] < keep))
    s = torch.einsum("bshd,bjhd->bhsj", q.double(), kk) * scale
    s = s - r1.double()[None, :, None, None] * torch.log1p(r2.double()[None, :, None, None] * d.clamp(min=0).double())
    w = s.masked_fill(~seen, float("-inf")).softmax(-1)
    return torch.einsum("hg,bgsj,bjhd->bshd", talk.double(), w, vv)


def _inputs(B, S, H, G, dim, vdim, window, keep, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g).to(dtype).cuda()
    proj = r(B * S, H * dim + G * dim + G * vdim)
    q, k, v = proj.split([H * dim, G * dim, G * vdim], 1)
    ring_k, ring_v = r(B, keep + window, G, dim), r(B, keep + window, G, vdim)
    r1, r2 = r(H).abs() + 0.1, r(H).abs() + 0.1
    talk = (torch.eye(H) + 0.2 * torch.randn(H, H, generator=g)).to(dtype).cuda()
    return proj, q.unflatten(0, (B, S)).unflatten(2, (H, dim)), k.unflatten(0, (B, S)).unflatten(2, (G, dim)), \
        v.unflatten(0, (B, S)).unflatten(2, (G, vdim)), ring_k, ring_v, r1, r2, talk


def _run(proj, q, k, v, ring_k, ring_v, r1, r2, talk, window, keep, pos0):
    """cd_window_attention_rows; q, k and v lie in the rows of proj."""
    from complexity_deep_b200 import _lib, ops
    (B, S, H, dim), G, vdim, dtype = q.shape, k.shape[2], v.shape[3], q.dtype
    ones = torch.ones(dim, dtype=dtype, device="cuda")
    out = torch.zeros(B * S, H * vdim, dtype=dtype, device="cuda")
    a = _lib.WindowAttn(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), ldp=proj.stride(0), q_w=ones.data_ptr(),
                        k_w=ones.data_ptr(), r1=r1.data_ptr(), r2=r2.data_ptr(), talk=talk.data_ptr(),
                        ring_k=ring_k.data_ptr(), ring_v=ring_v.data_ptr(), out=out.data_ptr(), ldo=out.stride(0),
                        pos_dev=None, scale=dim ** -0.5, eps=1e-6, out_scale=1.0, B=B, S=S, H=H, G=G, dim=dim, dp=dim,
                        vdim=vdim, vp=vdim, window=window, keep=keep, pos0=pos0, normed=1)
    assert _lib.load().cd_window_attention_rows(ctypes.byref(a), 1 if dtype == torch.float32 else 0, ops._stream()) == 0
    return out.view(B, S, H, vdim)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,S,H,G,dim,vdim,window,keep,pos0", [
    (16, 301, 6, 2, 48, 48, 300, 5, 0), (4, 1201, 12, 4, 32, 32, 130, 3, 0), (80, 5, 32, 8, 128, 128, 150, 2, 160),
    (2, 150, 16, 16, 128, 128, 200, 7, 230), (16, 130, 5, 5, 64, 32, 150, 1, 90), (2, 509, 8, 4, 128, 128, 512, 4, 0),
    (2, 160, 32, 2, 128, 128, 700, 0, 650), (1, 145, 8, 4, 128, 128, 512, 4, 700), (1, 145, 8, 4, 128, 128, 512, 4, 0), (80, 151, 20, 2, 16, 16, 90, 130, 128),
    (3, 60, 8, 4, 48, 64, 2, 4, 9)])
def test_tiles(B, S, H, G, dim, vdim, window, keep, pos0, dtype):
    proj, *x = _inputs(B, S, H, G, dim, vdim, window, keep, dtype, S + H)
    want = _reference(*x, window, keep, pos0, dim ** -0.5)
    got = _run(proj, *x, window, keep, pos0).double()
    bound = want.abs().amax((2, 3), keepdim=True) * 2e-6
    if dtype == torch.bfloat16:
        bound = bound + want.abs() * 2.0 ** -8
    assert bool(((got - want).abs() <= bound).all()), ((got - want).abs() / bound).max()


@pytest.mark.parametrize("what", ["query", "key", "bias"])
@pytest.mark.parametrize("S", [145, 401])
def test_nan_reaches_the_queries_that_see_it(S, what):
    """One query per cluster (145 tokens) and tiles (401) alike: a NaN score makes its query NaN, and no other one. The heads are
    mixed by a dense matrix, so a NaN in one of them is one in all."""
    H, G, dim, window, keep = 8, 4, 128, 256, 4
    proj, q, k, v, ring_k, ring_v, r1, r2, talk = _inputs(1, S, H, G, dim, dim, window, keep, torch.float32, S)
    clean = _run(proj, q, k, v, ring_k, ring_v, r1, r2, talk, window, keep, 0)[0]
    i, at = torch.arange(S, device="cuda"), 70                    # the third query of a tile
    if what == "query":
        q[0, at, 3, 5] = float("nan")
        hit = i == at
    elif what == "key":
        k[0, at, 2, 7] = float("nan")
        hit = (i >= at) & (i - at < window)
    else:
        r2[6] = -1.0 / 32.5                                       # log1p of less than -1 from a distance of 33 on
        hit = i >= 33
    got = _run(proj, q, k, v, ring_k, ring_v, r1, r2, talk, window, keep, 0)[0]
    assert bool(got[hit].isnan().all()) and bool(got[~hit].isfinite().all())
    if what != "bias":
        assert torch.equal(got[~hit], clean[~hit])


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("S", [145, 401])
def test_a_value_reaches_only_the_queries_that_see_it(S, bad):
    """Queries of a tile ahead of a key, or beyond its window, give it weight zero: infinities and NaN must not come through that."""
    H, G, dim, window, keep, at = 8, 4, 128, 256, 4, 70           # the third query of a tile, and the third beyond the window
    proj, q, k, v, ring_k, ring_v, r1, r2, talk = _inputs(1, S, H, G, dim, dim, window, keep, torch.float32, S)
    clean = _run(proj, q, k, v, ring_k, ring_v, r1, r2, talk, window, keep, 0)[0]
    v[0, at, 1, 9] = bad
    got = _run(proj, q, k, v, ring_k, ring_v, r1, r2, talk, window, keep, 0)[0]
    i = torch.arange(S, device="cuda")
    hit = torch.zeros_like(clean, dtype=torch.bool)
    hit[(i >= at) & (i - at < window), 2:4, 9] = True
    assert not bool(got[hit].isfinite().any()) and torch.equal(got[~hit], clean[~hit])
