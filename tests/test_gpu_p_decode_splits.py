"""Single-query attention over a cache (csrc/attention_decode.cu) where the rule that splits the rows over blocks
changes: one split, one more than a multiple of 48 rows, 32 and more splits' worth of rows, more pairs than one wave
holds; the length on the host and on the device (which must agree to the bit).

Tolerance against 64 bits on the same bf16 values: L exponentials and products in fp32, 2^-8 for the bf16 result, and
the hardware exponential's 2^-21 on weights that add up to one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,hkv,G,D,L", [(1, 1, 4, 64, 1), (1, 2, 1, 128, 48), (2, 1, 3, 64, 49), (1, 4, 3, 64, 302), (3, 2, 2, 128, 1537),
                                         (1, 1, 2, 64, 3300), (37, 8, 2, 128, 97), (38, 8, 1, 64, 600), (20, 8, 4, 128, 143)])
def test_splits(B, hkv, G, D, L):
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(B * 1000 + L)
    r = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)
    hq, cap = hkv * G, L + 70
    qkv, k, v = r(B, (hq + 2 * hkv) * D), r(B, hkv, cap, D), r(B, hkv, cap, D)
    q = qkv[:, : hq * D].double().view(B, hkv, G, D)
    s = torch.einsum("bhgd,bhld->bhgl", q, k[:, :, :L].double()) * D ** -0.5
    want = torch.einsum("bhgl,bhld->bhgd", s.softmax(-1), v[:, :, :L].double()).reshape(B, hq * D)
    cq, ck, cv = qkv.cuda(), k.cuda(), v.cuda()
    got = ops.decode_attention(cq, ck[:, :, :L], cv[:, :, :L], None, hq, hkv, D)
    assert bool(((got.double().cpu() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all())
    length = torch.tensor([L], dtype=torch.int32, device="cuda")
    # the capacity may ask for more splits than the length uses: the same split of the rows all the same
    assert torch.equal(ops.decode_attention(cq, ck, cv, None, hq, hkv, D, kv_len_dev=length), got)
