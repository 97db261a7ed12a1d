"""Chunked linear attention where a channel's thread has a segment of every length (eight threads a channel down to one, whose
64 decays do not all stay in registers) and where chunks end early: against the walk token by token of the same call in
fp32 storage of the same bf16 values.

The walk keeps fp32 throughout; the chunks round decayed operands to two bf16 parts (2^-17) and the result to bf16 (2^-9 of
its value). The head norm divides by the row's rms, so errors are measured against a row's largest value."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(dtype, S, B, H, dim, vdim, src, state):
    from complexity_deep_b200 import ops
    dkp, dvp, rank = -(-dim // 16) * 16, -(-vdim // 16) * 16, 16
    t = {k: v.to(dtype) for k, v in src.items()}
    widths = [H * dkp, H * dkp, H * dvp, H * dvp, rank]
    q, k, v, gate, inner = t["proj"].split(widths, 1)
    out = torch.zeros(B * S, H * dvp, dtype=dtype, device="cuda")
    ops.linear_attention_({"q": q, "k": k, "v": v, "gate": gate, "inner": inner}, out,
                          {"a2": t["a2"], "a2_b": t["a2_b"], "norm": t["norm"]}, state, batch=B, seq_len=S, heads=H, dim=dim,
                          vdim=vdim, tau=16.0, eps=1e-6, out_scale=0.7)
    return out


@pytest.mark.parametrize("dim,vdim", [(16, 16), (32, 128), (48, 64), (64, 256), (128, 128), (144, 32), (256, 64)])
@pytest.mark.parametrize("S", [16, 63, 64, 65, 200])
def test_segments(dim, vdim, S):
    B, H = 2, 3
    g = torch.Generator().manual_seed(dim + S)
    r = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).cuda()
    dkp, dvp, rank = dim, vdim, 16
    q = r(B * S, H * dkp)
    k = (0.6 * q + 0.8 * r(B * S, H * dkp)).to(torch.bfloat16)    # a token's own part of the result is not noise around zero
    src = {"proj": torch.cat([q, k, r(B * S, H * dvp), r(B * S, H * dvp), r(B * S, rank)], 1),
           "a2": 0.3 * r(H * dkp, rank), "a2_b": r(H * dkp), "norm": r(dvp).abs() + 0.5}
    start = torch.randn(B, H, dkp, dvp, generator=g).cuda()
    s16, s32 = start.clone(), start.clone()
    got = _call(torch.bfloat16, S, B, H, dim, vdim, src, s16).float().view(B * S, H, dvp)
    want = _call(torch.float32, S, B, H, dim, vdim, src, s32).view(B * S, H, dvp)
    scale = want.abs().amax(-1, keepdim=True)
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + scale * 2.0 ** -8).all())
    assert bool(((s16 - s32).abs() <= s32.abs().amax() * 2.0 ** -12).all())
