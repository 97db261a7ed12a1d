"""Kernels of decode steps where their split of the work changes with the number of tokens: norms of the fp32 stream with
four warps a row, rotary embedding with a token's heads dealt to warps, window attention with any number of splits up to
eight, linear attention with narrow column blocks and states of more rows than a thread holds at a time."""
import numpy as np
import pytest
import torch

from test_gpu_j_mixers import TOL, Window, _rel

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("dtype", [BF, F32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("rows,width,ldx", [(1, 513, 520), (2, 2048, 2048), (64, 2049, 2056), (296, 1000, 1000), (297, 1000, 1000),
                                            (5, 4096, 4096), (5, 4097, 4104), (33, 512, 512)])
def test_stream_norms(rows, width, ldx, dtype):
    """fp32 sums of `width` squares are off by at most width 2^-24, the result by a few roundings and its storage's."""
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(rows + width)
    x, w = torch.zeros(rows, ldx), torch.zeros(ldx)
    x[:, :width], w[:width] = 3 * torch.randn(rows, width, generator=g) + 0.5, torch.randn(width, generator=g)
    w = w.to(dtype)
    xd, wd = x.double()[:, :width], w.double()[:width]
    rel = 2.0 ** -8 if dtype == BF else (width + 16) * 2.0 ** -24
    for centred in (False, True):
        c = xd - xd.mean(-1, keepdim=True) if centred else xd
        want = c * torch.rsqrt(c.square().mean(-1, keepdim=True) + 1e-6) * (wd if centred else wd + 1.0)
        got = ops.layernorm_f32(x.cuda(), w.cuda(), 1e-6, width=width) if centred else ops.rmsnorm_f32(x.cuda(), w.cuda(), 1e-6, 1.0, width=width)
        got = got.double().cpu()
        assert bool(((got[:, :width] - want).abs() <= want.abs() * rel * 1.1 + 1e-5).all())
        if centred:
            assert not bool(got[:, width:].any())


@pytest.mark.parametrize("hq,hkv,D", [(12, 4, 64), (16, 8, 128), (3, 1, 16), (5, 5, 256), (40, 8, 128)])
def test_rotary_embedding_does_not_depend_on_the_number_of_tokens(hq, hkv, D):
    from complexity_deep_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(D)
    T, N = 600, (hq + 2 * hkv) * D
    qkv = torch.randn(T, N, device="cuda", generator=g).to(BF)
    qw, kw = (torch.randn(D, device="cuda", generator=g).to(BF) for _ in range(2))
    cos, sin = (torch.randn(64, D, device="cuda", generator=g) for _ in range(2))
    whole = ops.qk_norm_rope_(qkv.clone(), qw, kw, cos, sin, 1e-6, 1, 7, hq, hkv, D)
    for t in (1, 9, 591):
        assert torch.equal(ops.qk_norm_rope_(qkv[:t].clone(), qw, kw, cos, sin, 1e-6, 1, 7, hq, hkv, D), whole[:t])
    k, v = (torch.zeros(9, hkv, 64, D, dtype=BF, device="cuda") for _ in range(2))
    pos = torch.tensor([7], dtype=torch.int32, device="cuda")
    assert torch.equal(ops.decode_rope_append(qkv[:9].clone(), qw, kw, cos, sin, 1e-6, hq, hkv, D, k, v, pos), whole[:9])
    heads = whole[:9].view(9, -1, D)
    assert torch.equal(k[:, :, 7], heads[:, hq:hq + hkv]) and torch.equal(v[:, :, 7], heads[:, hq + hkv:])


@pytest.mark.parametrize("dtype", [BF, F32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("B,H,G,size,keep", [(148, 2, 1, 150, 3), (100, 1, 1, 195, 0), (44, 4, 2, 260, 4), (60, 2, 1, 340, 2),
                                             (1, 4, 1, 400, 5), (20, 5, 1, 300, 1), (63, 8, 8, 20, 1), (75, 12, 6, 24, 0)])
def test_window_decode_splits(B, H, G, size, keep, dtype):
    w = Window(dtype, size + keep + 6, H, G, 16, 16, size, keep, B, seed=B)
    assert _rel(w.run([w.T - 5] + [1] * 5), w.reference()) <= TOL[dtype]


@pytest.mark.parametrize("dtype", [BF, F32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("B,H,G,dim,vdim,size,keep", [(75, 4, 1, 72, 40, 127, 1), (37, 8, 2, 130, 16, 255, 1), (149, 2, 1, 40, 72, 64, 0),
                                                      (20, 5, 5, 200, 30, 129, 0)])
def test_window_decode_splits_by_what_an_sm_holds(B, H, G, dim, vdim, size, keep, dtype):
    """Kernels of which an SM holds one, two or three blocks: heads of each width, one to four query heads a block."""
    w = Window(dtype, size + keep + 3, H, G, dim, vdim, size, keep, B, seed=B)
    assert _rel(w.run([w.T - 2] + [1] * 2), w.reference()) <= TOL[dtype]


@pytest.mark.parametrize("B,H,dk,dv", [(1, 1, 160, 16), (2, 2, 48, 80), (40, 4, 32, 32), (3, 5, 272, 48), (80, 4, 128, 32), (1, 2, 512, 144),
                                       (74, 4, 144, 48), (75, 4, 144, 48), (99, 3, 32, 272)])
def test_linear_attention_forms_agree(B, H, dk, dv):
    """Token by token from a carried state (one kernel) and all tokens at once in 32 bits (another) against 64 bits."""
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(B * 7 + dk)
    T, rank = 19, 8
    r = lambda *s: torch.randn(*s, generator=g)
    q, k, v, gate = r(B, T, H * dk), r(B, T, H * dk), r(B, T, H * dv), r(B, T, H * dv)
    inner, a2, b2, norm = r(B, T, rank), r(H * dk, rank) * 0.3, r(H * dk), 1 + 0.1 * r(dv)
    decay = torch.nn.functional.logsigmoid(inner.double() @ a2.double().t() + b2.double()) / 16.0
    decay = decay.exp().view(B, T, H, dk)
    s, want = torch.zeros(B, H, dk, dv, dtype=torch.float64), torch.zeros(B, T, H, dv, dtype=torch.float64)
    for t in range(T):
        s = s * decay[:, t, ..., None] + k[:, t].double().view(B, H, dk, 1) * v[:, t].double().view(B, H, 1, dv)
        want[:, t] = (q[:, t].double().view(B, H, 1, dk) @ s)[:, :, 0] * dk ** -0.5
    want = want * torch.rsqrt(want.square().mean(-1, keepdim=True) + 1e-6) * norm.double()
    want = want.flatten(2) * torch.nn.functional.silu(gate.double())

    def run(lo, hi, state):
        n = hi - lo
        buf = torch.cat([x[:, lo:hi] for x in (q, k, v, gate, inner)], 2).reshape(B * n, -1).cuda()
        at, cols = 0, {}
        for name, width in (("q", H * dk), ("k", H * dk), ("v", H * dv), ("gate", H * dv), ("inner", rank)):
            cols[name] = buf[:, at:at + width]
            at += width
        out = torch.zeros(B * n, H * dv, device="cuda")
        call(cols, out, state, n)
        return out.double().cpu().view(B, n, -1)

    weights = {"a2": a2.cuda(), "a2_b": b2.cuda(), "norm": norm.cuda()}

    def call(cols, out, state, n):
        ops.linear_attention_(cols, out, weights, state, batch=B, seq_len=n, heads=H, dim=dk, vdim=dv, tau=16.0, eps=1e-6,
                              out_scale=1.0)

    whole_state, step_state = (torch.zeros(B, H, dk, dv, device="cuda") for _ in range(2))
    whole = run(0, T, whole_state)
    steps = torch.cat([run(t, t + 1, step_state) for t in range(T)], 1)
    for got in (whole, steps):
        assert float((got - want).abs().max()) <= 2e-4 * float(want.abs().max())
    for state in (whole_state, step_state):
        assert float((state.double().cpu() - s).abs().max()) <= 1e-5 * float(s.abs().max())
