"""Window attention of one token per sequence (cd_window_attention_decode) on both sides of the rule that says where the heads are mixed:
beside the values, or by a kernel between scores and values. Heads of their own keys and shared ones, more keys a block than it
mixes at a time, more blocks than one wave. Against 64 bits; tolerances as in test_gpu_y_window_tiles.py, with 2^-7 for a
bf16 norm of query and key, and 2^-18 for the exponential of bf16 storage."""
import ctypes

import pytest
import torch

from test_gpu_y_window_tiles import _inputs, _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,G,dim,window,dtype,kernels", [
    (1, 16, 8, 64, 4100, torch.bfloat16, 3), (4, 16, 8, 64, 1028, torch.bfloat16, 2), (1, 32, 32, 64, 520, torch.bfloat16, 2),
    (1, 6, 2, 128, 4099, torch.bfloat16, 3), (2, 16, 16, 64, 2052, torch.float32, 3), (8, 16, 16, 64, 516, torch.float32, 2),
    (4, 8, 8, 32, 516, torch.float32, 3), (1, 64, 64, 32, 1030, torch.float32, 2), (2, 96, 96, 16, 2052, torch.float32, 3),
    (100, 8, 4, 64, 300, torch.float32, 3), (3, 40, 5, 32, 77, torch.float32, 2)])
def test_mixing(B, H, G, dim, window, dtype, kernels):
    from complexity_deep_b200 import _lib, ops
    lib, keep, pos0, fp32 = _lib.load(), 3, window + 50, 1 if dtype == torch.float32 else 0
    proj, q, k, v, ring_k, ring_v, r1, r2, talk = _inputs(B, 1, H, G, dim, dim, window, keep, dtype, H + window)
    norm = lambda t: (t.double() * torch.rsqrt(t.double().square().mean(-1, keepdim=True) + 1e-6)).to(dtype)
    want = _reference(norm(q), norm(k), v, ring_k, ring_v, r1, r2, talk, window, keep, pos0, dim ** -0.5)
    ones = torch.ones(dim, dtype=dtype, device="cuda")
    out = torch.zeros(B, H * dim, dtype=dtype, device="cuda")
    a = _lib.WindowAttn(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), ldp=proj.stride(0), q_w=ones.data_ptr(), k_w=ones.data_ptr(),
                        r1=r1.data_ptr(), r2=r2.data_ptr(), talk=talk.data_ptr(), ring_k=ring_k.data_ptr(), ring_v=ring_v.data_ptr(),
                        out=out.data_ptr(), ldo=out.stride(0), pos_dev=None, scale=dim ** -0.5, eps=1e-6, out_scale=1.0, B=B, S=1, H=H,
                        G=G, dim=dim, dp=dim, vdim=dim, vp=dim, window=window, keep=keep, pos0=pos0, normed=0)
    n = lib.cd_window_attention_decode_workspace_bytes(ctypes.byref(a))
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    assert lib.cd_window_attention_decode_launches(ctypes.byref(a), fp32) == kernels
    assert lib.cd_window_attention_decode(ctypes.byref(a), ws.data_ptr(), n, fp32, ops._stream()) == 0
    got = out.view(B, 1, H, dim).double()
    bound = want.abs().amax((2, 3), keepdim=True) * (2e-6 if fp32 else 2.0 ** -7)
    if not fp32:
        bound = bound + want.abs() * 2.0 ** -8
    assert bool(((got - want).abs() <= bound).all()), ((got - want).abs() / bound).max()
