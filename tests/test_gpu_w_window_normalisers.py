"""Window attention of prompts with the normalisers found by a kernel of their own against the form without a workspace,
which finds them in a first pass over the keys: rows around the tiles of 128 keys and queries and their halves, windows smaller
than a warp's 32 queries, kept tokens on both sides of a tile, portions whose earlier keys come from the ring, one and
several query heads a key head, head widths that fill no 128 columns.

Both sum the same fp32 exponentials in another order: 2^-20 on a normaliser, which moves a weight by as much before it is
rounded to two bf16 parts (2^-17), and the mixed weights round to bf16: a result may differ by one unit of its last place."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(B, S, H, G, dim, vdim, window, keep, pos0):
    from complexity_deep_b200 import _lib, ops
    lib = _lib.load()
    g = torch.Generator().manual_seed(S + 31 * H + window)
    r = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).cuda()
    dp, vp = -(-dim // 16) * 16, -(-vdim // 16) * 16

    def heads(rows, n, used, width):
        t = r(rows, n, width)
        t[..., used:] = 0
        return t.reshape(rows, n * width)
    proj = torch.cat([heads(B * S, H, dim, dp), heads(B * S, G, dim, dp), heads(B * S, G, vdim, vp)], 1)
    q, k, v = proj.split([H * dp, G * dp, G * vp], 1)
    ring_k = heads(B * (keep + window), G, dim, dp)
    ring_v = heads(B * (keep + window), G, vdim, vp)
    r1, r2 = r(H).abs() + 0.1, r(H).abs() + 0.1
    talk = (torch.eye(H) + 0.2 * torch.randn(H, H, generator=g)).to(torch.bfloat16).cuda()
    ones = torch.ones(dp, dtype=torch.bfloat16, device="cuda")
    outs = []
    for own in (False, True):
        out = torch.zeros(B * S, H * vp, dtype=torch.bfloat16, device="cuda")
        a = _lib.WindowAttn(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), ldp=proj.stride(0), q_w=ones.data_ptr(),
                            k_w=ones.data_ptr(), r1=r1.data_ptr(), r2=r2.data_ptr(), talk=talk.data_ptr(),
                            ring_k=ring_k.data_ptr(), ring_v=ring_v.data_ptr(), out=out.data_ptr(), ldo=out.stride(0),
                            pos_dev=None, scale=dim ** -0.5, eps=1e-6, out_scale=0.7, B=B, S=S, H=H, G=G, dim=dim, dp=dp,
                            vdim=vdim, vp=vp, window=window, keep=keep, pos0=pos0, normed=1)
        ref = ctypes.byref(a)
        assert lib.cd_window_attention_prefill_supported(ref)
        if own:
            n = lib.cd_window_attention_prefill_workspace_bytes(ref)
            assert n == 4 * B * H * S
            ws = torch.full((n // 4,), float("nan"), device="cuda")
            assert lib.cd_window_attention_prefill_ws(ref, ws.data_ptr(), n - 4, ops._stream()) == 1
            assert lib.cd_window_attention_prefill_ws(ref, ws.data_ptr(), n, ops._stream()) == 0
            torch.cuda.synchronize()
            assert bool(ws.isfinite().all())
        else:
            assert lib.cd_window_attention_prefill(ref, ops._stream()) == 0
        outs.append(out.float())
    ops.status_fetch()
    want, got = outs
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -7 + 2.0 ** -9).all())


@pytest.mark.parametrize("S", [2, 15, 16, 17, 63, 64, 65, 127, 128, 129, 200, 513])
def test_rows(S):
    _run(2, S, 16, 8, 128, 128, 96, 4, 0)


@pytest.mark.parametrize("B,S,H,G,dim,vdim,window,keep,pos0", [
    (1, 70, 6, 2, 40, 56, 300, 5, 0), (1, 150, 8, 4, 128, 128, 512, 4, 450), (2, 33, 8, 8, 64, 64, 5, 70, 200),
    (1, 300, 16, 4, 128, 64, 1, 0, 17), (1, 260, 4, 1, 16, 16, 130, 64, 1000), (3, 129, 16, 16, 112, 128, 40, 65, 39),
    (1, 1100, 16, 8, 128, 128, 1024, 4, 0)])
def test_windows_and_portions(B, S, H, G, dim, vdim, window, keep, pos0):
    _run(B, S, H, G, dim, vdim, window, keep, pos0)
