"""The kernel for products of few rows (csrc/gemm_few_rows.cu) through its entry points, at the edges of its blocks
(8 rows, 16 / 32 weight rows, steps of 32 along K), against 64-bit products of the same bf16 values.

Tolerance: K products summed in fp32 in some order are off by at most (K + 16) 2^-23 sum |x| |w|, a bf16 result by
another 2^-8 of its size."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _rand(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g) * scale).to(BF)


def _near(got, want, slack, bits=8):
    got, want = got.double().cpu(), want.double()
    err = (got - want).abs()
    bound = slack + want.abs() * 2.0 ** -bits + 1e-30
    assert bool((err <= bound).all()), float((err / bound).max())


def _product(x, w):
    """x w^T in 64 bits and the bound on an fp32 sum of it"""
    x, w = x.double(), w.double()
    return x @ w.t(), (x.abs() @ w.abs().t()) * ((x.shape[1] + 16) * 2.0 ** -23)


ROWS = [1, 7, 8, 9, 16, 17, 32, 33, 48, 49, 64]


@pytest.mark.parametrize("T,K,N", [(t, k, n) for t, (k, n) in zip(ROWS, [
    (8, 8), (40, 24), (72, 40), (768, 264), (1032, 16), (96, 32), (2048, 2056), (264, 1280), (32, 48), (520, 72), (64, 9504)])]
    + [(17, 264, 264), (48, 776, 776), (64, 40, 40)]                                  # square: mu_proj as well
    + [(1, 72, 9480), (8, 64, 9496), (9, 40, 9448), (17, 72, 9512), (33, 24, 9480)])   # 32 weight rows a block, the last not full
def test_store_epilogues(T, K, N):
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(T * 1000 + N)
    x, w, mu, wm = _rand(g, T, K), _rand(g, N, K), _rand(g, T, K), _rand(g, N, K)
    hi, lo = _rand(g, T, N, scale=4.0), _rand(g, T, N, scale=0.01)
    y, slack = _product(x, w)
    cx, cw = x.cuda(), w.cuda()
    _near(ops.linear(cx, cw), y, slack)
    _near(ops.linear(cx, cw, hi.cuda()), y + hi.double(), slack + hi.abs().double() * 2.0 ** -22)
    a, b = ops.linear(cx, cw, hi.cuda(), residual_lo=lo.cuda(), want_lo=True)
    full = y + hi.double() + lo.double()
    _near(a, full, slack + hi.abs().double() * 2.0 ** -22)
    _near(a.double().cpu() + b.double().cpu(), full, slack + hi.abs().double() * 2.0 ** -22, bits=15)
    _near(ops.project(cx, cw, act="relu2"), y.clamp(min=0) ** 2, 2 * y.abs() * slack + slack ** 2)
    z, more = _product(mu, wm)
    _near(ops.mu_qkv(cx, mu.cuda(), cw, wm.cuda()), y + z, slack + more)
    scale, res = _rand(g, N), torch.randn(T, N, generator=g)
    f = ops.linear_to_f32(cx, cw, residual=res.cuda(), col_scale=scale.cuda(), scale=0.75)
    s = 0.75 * scale.double()
    _near(f, res.double() + s * y, (slack + y.abs() * 2.0 ** -22) * s.abs() + res.abs().double() * 2.0 ** -22, bits=23)
    wide = torch.full((T, K + 16), float("nan"), dtype=BF)      # rows that lie apart
    wide[:, 8: 8 + K] = x
    _near(ops.project(wide.cuda()[:, 8: 8 + K], cw), y, slack)
    if N == K:
        _near(ops.mu_proj(cx, cw, scale.cuda(), -0.5, 0.5, out_clamp=(-1.0, 1.0)),
              (y + scale.double().clamp(-0.5, 0.5)).clamp(-1.0, 1.0), slack)
    ops.status_fetch()


@pytest.mark.parametrize("counts,H,I,bn,shared", [
    ([1, 0, 2], 40, 24, 32, 40), ([0, 9, 17, 0, 33], 72, 104, 64, 0), ([8, 8, 0, 16, 32], 264, 136, 128, 72),
    ([0] * 30 + [40, 1], 104, 200, 256, 0), ([5] + [0] * 63, 64, 48, 64, 0), ([3, 61], 520, 344, 256, 128)])
def test_row_groups(counts, H, I, bn, shared):
    check_row_groups(counts, H, I, bn, shared, 0)


def check_row_groups(counts, H, I, bn, shared, most):
    """Groups of experts, empty ones among them: both gated units, the down projection with its scattered rows, its
    residual pair and a shared expert."""
    from complexity_deep_b200 import ops
    T, E = sum(counts), len(counts)
    g = torch.Generator().manual_seed(T * 100 + H)
    seg = torch.tensor([0] + counts).cumsum(0).int()
    x = _rand(g, T, H)
    gate, up, down = _rand(g, E, I, H, scale=0.1), _rand(g, E, I, H, scale=0.1), _rand(g, E, H, I, scale=0.1)
    packed = ops.pack_gate_up(gate.cuda(), up.cuda(), bn)
    cx, cseg = x.cuda(), seg.cuda()
    sides = [(_product(x[a:b], gate[e]), _product(x[a:b], up[e])) for e, (a, b) in enumerate(zip(seg[:-1], seg[1:]))]
    (gv, gs), (uv, us) = (tuple(torch.cat([s[i][j] for s in sides]) for j in (0, 1)) for i in (0, 1))
    slack = gs * (uv.abs() + us) * 1.1 + us * gv.abs() + (gv * uv).abs() * 2.0 ** -19
    _near(ops.moe_up(cx, cseg, E, packed, I, bn), F.silu(gv) * uv, slack)
    limit, alpha = 1.5, 1.702
    lg, lu = gv.clamp(max=limit), uv.clamp(-limit, limit)
    _near(ops.glu_up(cx, packed, I, bn, alpha, limit, 1.0, seg_offsets=cseg, most_rows=most), lg * torch.sigmoid(alpha * lg) * (lu + 1.0),
          2 * gs * (limit + 1) + us * limit + (lg * (lu + 1)).abs() * 2.0 ** -19 + 1e-6)
    h = _rand(g, T, I)
    rows = torch.randperm(T, generator=g).int()
    hi, lo = _rand(g, T, H, scale=4.0), _rand(g, T, H, scale=0.01)
    parts = [_product(h[a:b], down[e]) for e, (a, b) in enumerate(zip(seg[:-1], seg[1:]))]
    y, s = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
    hs = ws = None
    if shared:
        hs, ws = _rand(g, T, shared), _rand(g, H, shared, scale=0.1)
        z, more = _product(hs, ws)
        y, s = y + z, s + more
        hs, ws = hs.cuda(), ws.cuda()
    want, bound = torch.zeros(T, H, dtype=torch.float64), torch.zeros(T, H, dtype=torch.float64)
    want[rows.long()], bound[rows.long()] = y, s
    a, b = ops.moe_down(h.cuda(), down.cuda(), hs, ws, cseg, E, rows.cuda(), hi.cuda(), residual_lo=lo.cuda(), want_lo=True,
                        most_rows=most)
    want = want + hi.double() + lo.double()
    bound = bound + hi.abs().double() * 2.0 ** -21
    _near(a, want, bound)
    _near(a.double().cpu() + b.double().cpu(), want, bound, bits=15)
    ops.status_fetch()


def test_rows_do_not_depend_on_their_neighbours():
    """A row's result has the same bits whatever rows are computed with it (the order of the sums is that of K alone)."""
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(3)
    x, w = _rand(g, 64, 776).cuda(), _rand(g, 1288, 776).cuda()
    full = ops.linear(x, w)
    for n in (1, 8, 9, 20, 33, 50):
        assert torch.equal(ops.linear(x[:n].contiguous(), w), full[:n]), n


@pytest.mark.parametrize("rows,I,Is,bn,bn_s", [(1, 40, 104, 32, 256), (17, 136, 24, 256, 32), (64, 200, 328, 64, 128)])
def test_routed_and_shared_weights_of_two_layouts(rows, I, Is, bn, bn_s):
    """In one launch the bits of the same weights packed alike; calls of more than 64 rows refuse two layouts."""
    from complexity_deep_b200 import ops
    E, H = 4, 72
    g = torch.Generator().manual_seed(rows)
    x = _rand(g, 65, H).cuda()
    seg = torch.tensor([0, rows // 3, rows // 3, rows - rows // 2, rows], dtype=torch.int32).cuda()
    gate, up, sg, su = (_rand(g, *s, scale=0.1).cuda() for s in ((E, I, H), (E, I, H), (1, Is, H), (1, Is, H)))
    routed, shared = ops.pack_gate_up(gate, up, bn), ops.pack_gate_up(sg, su, bn_s)
    got = ops.moe_up_pair(x[:rows], seg, E, routed, I, shared, Is, bn, bn_s)
    want = ops.moe_up_pair(x[:rows], seg, E, routed, I, ops.pack_gate_up(sg, su, bn), Is, bn)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    whole = torch.tensor([0, 65, 65, 65, 65], dtype=torch.int32).cuda()
    with pytest.raises(RuntimeError):
        ops.moe_up_pair(x, whole, E, routed, I, shared, Is, bn, bn_s)


def test_a_layer_packs_its_shared_expert_once_for_decoding_and_short_prompts():
    from complexity_deep_b200 import ops
    from complexity_deep_b200.core.token_routed_mlp import TokenRoutedMLP
    mlp = TokenRoutedMLP(hidden_size=768, intermediate_size=2816, num_experts=4, vocab_size=100).to("cuda", BF)
    assert len({ops.choose_block_n(mlp.shared_gate.weight.shape[0], n) for n in (1, 64, 100)}) == 1
    assert ops.choose_block_n(mlp.expert_intermediate_size, 1, 4) != ops.choose_block_n(mlp.shared_gate.weight.shape[0], 1)
    with torch.no_grad():
        for n in (1, 64, 100):
            mlp(torch.zeros(1, n, 768, dtype=BF, device="cuda"), torch.zeros(1, n, dtype=torch.long, device="cuda"))
    assert sum(name.startswith("shared_gate_up") for name in mlp._derived._slots) == 1
