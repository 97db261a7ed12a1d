"""The 32-bit matrix product (csrc/linear_f32.cu) through its entry points, at the edges of each of its tiles.

Tolerance: a chain of K fused multiply-adds is off by at most K 2^-24 sum |x| |w| (1 + tiny), scale, column factor and
residual by one rounding each. Every output is one chain over k, whatever the tile, so that a row by itself and the
same row among many (which take other tiles) agree to the bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


def _near(got, want, slack):
    err = (got.double().cpu() - want).abs()
    assert bool((err <= slack + 1e-30).all()), float((err / (slack + 1e-30)).max())


@pytest.mark.parametrize("T,K,N", [(1, 4, 1), (15, 36, 31), (17, 1024, 33), (8, 40, 19204), (33, 72, 2052), (65, 100, 4100),
                                   (127, 20, 1030), (200, 516, 1024), (500, 64, 1000), (1018, 256, 1028), (1025, 28, 4132),
                                   (1000, 16, 17000)])
def test_dense(T, K, N):
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(T + 7 * N)
    wide = torch.full((T, K + 8), float("nan"))                      # rows that lie apart
    wide[:, 4: 4 + K] = torch.randn(T, K, generator=g)
    w, res, col = torch.randn(N, K, generator=g), torch.randn(T, N, generator=g), torch.randn(N, generator=g)
    x = wide[:, 4: 4 + K].double()
    y, mag = x @ w.double().t(), (x.abs() @ w.double().abs().t()) * (K + 2) * U
    cx, cw = wide.cuda()[:, 4: 4 + K], w.cuda()
    plain = ops.project(cx, cw)
    _near(plain, y, mag)
    _near(ops.project(cx, cw, act="relu2"), y.clamp(min=0) ** 2, 2 * y.abs() * mag + mag ** 2 + y ** 2 * 2 * U)
    s = 0.75 * col.double()
    got = ops.linear_to_f32(cx, cw, residual=res.cuda(), col_scale=col.cuda(), scale=0.75)
    _near(got, res.double() + s * y, (mag + 4 * U * y.abs()) * s.abs() + (res.double().abs() + (s * y).abs()) * 2 * U)
    for t in (0, T // 2, T - 1):
        assert torch.equal(ops.project(cx[t: t + 1], cw)[0], plain[t])


@pytest.mark.parametrize("counts,K,N", [([0, 3, 0, 130], 36, 100), ([17] * 12, 200, 2000), ([1] + [0] * 31, 64, 48),
                                        ([700, 65, 1], 24, 1408)])
def test_row_groups(counts, K, N):
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(sum(counts))
    T, seg = sum(counts), torch.tensor([0] + counts).cumsum(0).int()
    x, w = torch.randn(T, K, generator=g), torch.randn(len(counts), N, K, generator=g)
    got = ops.grouped_linear_f32(x.cuda(), w.cuda(), seg.cuda(), "test")
    for e, (a, b) in enumerate(zip(seg[:-1], seg[1:])):
        xd, wd = x[a:b].double(), w[e].double()
        _near(got[a:b], xd @ wd.t(), (xd.abs() @ wd.abs().t()) * (K + 2) * U)


@pytest.mark.parametrize("T,K,N", [(5, 40, 31), (130, 64, 1000), (600, 24, 1028), (7, 516, 66)])
def test_factors_and_residual_round_as_one_multiply_add(T, K, N):
    """Behind the sum come the scale, the column factor and the residual; the last factor and the residual round once,
    whether the columns are stored by fours or singly. 80-bit numbers hold the product exactly."""
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(T + N)
    x, w = torch.randn(T, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    res, col = torch.randn(T, N, generator=g), torch.randn(N, generator=g)
    y, scale = ops.project(x, w).cpu().numpy(), np.float32(0.7)
    wide = lambda a: a.numpy().astype(np.longdouble)
    for c in (None, col):
        first, last = (y, np.longdouble(scale)) if c is None else (y * scale, wide(c))
        want = first.astype(np.longdouble) * last
        got = ops.linear_to_f32(x, w, residual=res.cuda(), col_scale=None if c is None else c.cuda(), scale=0.7)
        assert np.array_equal(got.cpu().numpy(), (want + wide(res)).astype(np.float32))
        got = ops.linear_to_f32(x, w, col_scale=None if c is None else c.cuda(), scale=0.7)
        assert np.array_equal(got.cpu().numpy(), want.astype(np.float32))
