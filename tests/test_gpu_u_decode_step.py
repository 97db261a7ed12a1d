"""A decode step's attention in one launch (cd_decode_step_attention) against the two calls that it stands for: rotation
and append, then attention over the cache.  Every cluster size that csrc/decode_split.h gives (one to eight blocks a pair, 13 and
16), lengths far below the capacity that a launch is sized for, caches of several thousand rows, the new row first, last
and in the middle of a block's rows, caches with strides of their own, a position outside the cache (nothing is written),
tables and weights off a 16-byte boundary (the two calls run).

Both round q and k to bf16 after the same arithmetic, so the caches must agree to the bit and the result to two units of
bf16's last place (a fused multiply-add may be contracted differently)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(B, hkv, G, D, cap, norm, seed):
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).cuda()
    ang = torch.rand(cap, D // 2, generator=g) * 6
    ang = torch.cat([ang, ang], 1)
    w = (r(D), r(D)) if norm else (None, None)
    return r(B, (G + 2) * hkv * D), r(B, hkv, cap, D), r(B, hkv, cap, D), ang.cos().cuda(), ang.sin().cuda(), w


def _check(B, hkv, G, D, cap, pos, length, norm=True, token_major=False):
    from complexity_deep_b200 import ops
    qkv, k, v, cos, sin, (qw, kw) = _inputs(B, hkv, G, D, cap, norm, B + 7 * pos + cap)
    if token_major:                                      # same values, another order in memory
        k, v = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (k, v))
    state = torch.tensor([pos, length], dtype=torch.int32, device="cuda")
    hq = hkv * G
    k1, v1 = k.clone(memory_format=torch.preserve_format), v.clone(memory_format=torch.preserve_format)
    rot = ops.decode_rope_append(qkv.clone(), qw, kw, cos, sin, 1e-6, hq, hkv, D, k1, v1, state[:1])
    want = ops.decode_attention(rot, k1, v1, None, hq, hkv, D, kv_len_dev=state[1:])
    before = qkv.clone()
    got = ops.decode_step_attention(qkv, qw, kw, cos, sin, 1e-6, hq, hkv, D, k, v, state[:1], state[1:])
    assert torch.equal(qkv, before) and torch.equal(k, k1) and torch.equal(v, v1)
    # two units of the last place, or what a bf16 unit of q or k moves a score by (2^-8 of at most ~6)
    assert bool(((got.float() - want.float()).abs() <= want.float().abs() * 2.0 ** -7 + 2.0 ** -7).all())
    if pos + 1 == length:                                # against 64 bits on the rotated rows
        q = rot[:, : hq * D].double().view(B, hkv, G, D)
        s = torch.einsum("bhgd,bhld->bhgl", q, k1[:, :, :length].double()) * D ** -0.5
        ref = torch.einsum("bhgl,bhld->bhgd", s.softmax(-1), v1[:, :, :length].double()).reshape(B, hq * D)
        assert bool(((got.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 2.0 ** -8).all())


# one to eight blocks of 48 rows; 16 blocks of a pair (up to eight pairs) of 80 and of 144 rows, 13 (up to 24 pairs) of 80 and of 96;
# eight just below both
@pytest.mark.parametrize("B,hkv,G,D,cap", [(1, 2, 2, 64, 48 * n) for n in range(1, 9)] + [
    (1, 2, 2, 64, 1151), (1, 2, 2, 64, 1280), (2, 4, 1, 128, 2300), (1, 4, 3, 64, 2064), (2, 8, 2, 128, 935), (2, 8, 2, 128, 1040),
    (3, 8, 2, 64, 1248), (1, 12, 4, 64, 937)])
def test_cluster_sizes(B, hkv, G, D, cap):
    _check(B, hkv, G, D, cap, cap - 1, cap)


@pytest.mark.parametrize("length", [1, 16, 47, 385, 900, 1152, 1500, 4000])
def test_lengths_below_the_capacity(length):
    _check(1, 4, 2, 128, 4096, length - 1, length)
    _check(2, 8, 3, 64, 4096, length - 1, length)


@pytest.mark.parametrize("B,hkv,G,D,cap,pos", [(1, 2, 3, 64, 9000, 8999), (1, 8, 2, 128, 8200, 5000), (4, 8, 2, 128, 4100, 4099), (40, 8, 1, 64, 3000, 2999)])
def test_long_caches(B, hkv, G, D, cap, pos):
    _check(B, hkv, G, D, cap, pos, pos + 1)


@pytest.mark.parametrize("B,hkv,G,D,cap,pos", [(1, 4, 3, 64, 320, 0), (1, 4, 3, 64, 320, 16), (1, 4, 3, 64, 320, 47), (2, 1, 4, 128, 700, 699),
                                               (3, 2, 1, 128, 130, 64), (32, 8, 2, 128, 300, 255), (40, 8, 2, 64, 520, 519),
                                               (64, 8, 1, 128, 1100, 1023)])
def test_positions(B, hkv, G, D, cap, pos):
    for norm in (True, False):
        _check(B, hkv, G, D, cap, pos, pos + 1, norm, token_major=pos % 2 == 1)


@pytest.mark.parametrize("pos,length", [(-1, 40), (200, 200), (130, 60), (5, 0), (10, 190)])
def test_position_outside_the_rows_attended(pos, length):
    _check(2, 2, 2, 64, 200, pos, length)


@pytest.mark.parametrize("B,hkv,G,D,cap", [(1, 8, 2, 128, 9000), (2, 8, 1, 64, 4200), (1, 2, 4, 128, 6200), (4, 8, 2, 64, 8300), (1, 30, 1, 64, 8200)])
def test_a_length_below_the_capacity_gives_the_bits_of_a_launch_of_that_length(B, hkv, G, D, cap):
    """One cluster a pair, and several whose sums are added by a kernel behind them."""
    from complexity_deep_b200 import _lib, ops
    assert _lib.load().cd_decode_attention_workspace_bytes(B, hkv * G, hkv, cap, D) > 0
    qkv, k, v, *_ = _inputs(B, hkv, G, D, cap, False, cap)
    for length in (1, 300, 1500, 4095, 4096, cap - 1, cap):
        state = torch.tensor([length], dtype=torch.int32, device="cuda")
        got = ops.decode_attention(qkv, k, v, None, hkv * G, hkv, D, kv_len_dev=state)
        want = ops.decode_attention(qkv, k[:, :, :length], v[:, :, :length], None, hkv * G, hkv, D)
        assert torch.equal(got, want), length


@pytest.mark.parametrize("what", ["cos", "weight"])
def test_off_a_16_byte_boundary(what):
    from complexity_deep_b200 import ops
    B, hkv, G, D, cap, pos = 2, 2, 2, 64, 200, 77
    qkv, k, v, cos, sin, (qw, kw) = _inputs(B, hkv, G, D, cap, True, 5)
    state = torch.tensor([pos, pos + 1], dtype=torch.int32, device="cuda")
    k1, v1 = k.clone(), v.clone()
    want = ops.decode_step_attention(qkv, qw, kw, cos, sin, 1e-6, hkv * G, hkv, D, k1, v1, state[:1], state[1:])
    move = lambda t: torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)      # the same values one element further on
    if what == "cos":
        cos = move(cos)
    else:
        qw = move(qw)
    before = qkv.clone()
    got = ops.decode_step_attention(qkv, qw, kw, cos, sin, 1e-6, hkv * G, hkv, D, k, v, state[:1], state[1:])
    assert torch.equal(k, k1) and torch.equal(v, v1) and torch.equal(qkv, before)
    # what a rounding of q to bf16 moves a score by (2^-8 of at most ~6), as above
    assert bool(((got.float() - want.float()).abs() <= want.float().abs() * 2.0 ** -7 + 2.0 ** -7).all())


@pytest.mark.parametrize("B,hkv,G,D,cap", [(1, 2, 2, 64, 300), (2, 8, 2, 128, 1100), (64, 8, 1, 64, 700)])
def test_nan_and_infinities(B, hkv, G, D, cap):
    """A NaN score makes its head NaN and no other one; an infinite value its column; a row that sees nothing is zero."""
    from complexity_deep_b200 import ops
    hq, (qkv, k, v, cos, sin, (qw, kw)) = hkv * G, _inputs(B, hkv, G, D, cap, True, 11)
    run = lambda k, v, m=None: ops.decode_attention(qkv, k, v, m, hq, hkv, D).view(B, hkv, G, D)
    clean = run(k, v)
    assert bool(clean.isfinite().all())
    bad, worse = k.clone(), v.clone()
    bad[0, 1, cap - 2, 3] = float("nan")
    worse[0, 0, 5, 7] = float("inf")
    hit = torch.zeros_like(clean, dtype=torch.bool)
    hit[0, 1] = hit[0, 0, :, 7] = True
    got = run(bad, worse)
    assert bool(got[0, 1].isnan().all()) and not bool(got[hit].isfinite().any()) and torch.equal(got[~hit], clean[~hit])
    state = torch.tensor([cap - 1, cap], dtype=torch.int32, device="cuda")
    step = ops.decode_step_attention(qkv, qw, kw, cos, sin, 1e-6, hq, hkv, D, bad, worse, state[:1], state[1:]).view(B, hkv, G, D)
    assert bool(step[0, 1].isnan().all()) and not bool(step[hit].isfinite().any()) and bool(step[~hit].isfinite().all())
    mask = torch.full((1, 1, 1, cap), float("-inf"), dtype=torch.bfloat16, device="cuda")
    assert not bool(run(k, v, mask).any())
