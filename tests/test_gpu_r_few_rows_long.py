"""Products of few rows in the forms that other tests do not reach (csrc/gemm_few_rows.cu): sixteen shares of a long K (of up to 32 rows a warp each, of more two a
warp, and of row groups), K segments that end within a step or meet within a share, row groups in several waves of blocks. Against 64-bit products of the same bf16 values;
tolerances as in test_gpu_n_few_rows.py."""
import pytest
import torch

from test_gpu_n_few_rows import _near, _product, _rand, check_row_groups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("K,N", [(2048, 600), (2040, 1032), (2056, 2360), (4104, 592), (2016, 600)])
def test_long_k(T, K, N):
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(T * 100 + K)
    x, w, res = _rand(g, T, K), _rand(g, N, K), _rand(g, T, N)
    y, slack = _product(x, w)
    _near(ops.linear(x.cuda(), w.cuda(), res.cuda()), y + res.double(), slack + res.abs().double() * 2.0 ** -22)
    r32 = torch.randn(T, N, generator=g)
    _near(ops.linear_to_f32(x.cuda(), w.cuda(), residual=r32.cuda()), r32.double() + y, slack + r32.abs().double() * 2.0 ** -22, bits=23)


@pytest.mark.parametrize("T,K,N", [(1, 1032, 600), (9, 1096, 1032), (32, 2056, 640), (40, 1064, 600), (3, 520, 72)])
def test_two_segments(T, K, N):
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(T + K)
    x, w, mu, wm = _rand(g, T, K), _rand(g, N, K), _rand(g, T, K), _rand(g, N, K)
    (y, a), (z, b) = _product(x, w), _product(mu, wm)
    _near(ops.mu_qkv(x.cuda(), mu.cuda(), w.cuda(), wm.cuda()), y + z, a + b)


@pytest.mark.parametrize("counts,H,I", [([20, 0, 33, 11], 256, 2048), ([3, 0, 8, 9, 16, 1] * 8, 200, 704), ([0] * 63 + [33], 72, 712), ([8] * 64, 264, 392)])
def test_row_groups_in_several_waves(counts, H, I):
    check_row_groups(counts, H, I, 64, 0, 64)


def test_long_k_rows_do_not_depend_on_their_neighbours():
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(9)
    for K, N in ((2304, 1288), (2024, 1032)):              # the second: 64 steps, the least that is cut into sixteen
        x, w = _rand(g, 64, K).cuda(), _rand(g, N, K).cuda()
        full = ops.linear(x, w)
        for n in (1, 8, 9, 17, 32, 33, 48, 49):
            assert torch.equal(ops.linear(x[:n].contiguous(), w), full[:n]), (K, n)
    x, mu, w, wm = _rand(g, 64, 1032).cuda(), _rand(g, 64, 1032).cuda(), _rand(g, 1032, 1032).cuda(), _rand(g, 1032, 1032).cuda()
    full = ops.mu_qkv(x, mu, w, wm)                        # two segments, 66 steps together
    for n in (5, 32, 33):
        assert torch.equal(ops.mu_qkv(x[:n].contiguous(), mu[:n].contiguous(), w, wm), full[:n]), n


def test_long_k_rows_of_groups_do_not_depend_on_other_groups():
    """Down projections of row groups, K in sixteen shares: the first rows of each group alone and among more of them."""
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(10)
    E, H, I, few, many = 4, 256, 2048, [7, 9, 0, 13], [7, 30, 3, 24]
    w = _rand(g, E, H, I, scale=0.1).cuda()
    h = [_rand(g, n, I) for n in many]

    def run(counts):
        seg = torch.tensor([0] + counts).cumsum(0).int().cuda()
        x, T = torch.cat([a[:n] for a, n in zip(h, counts)]).cuda(), sum(counts)
        out = ops.moe_down(x, w, None, None, seg, E, torch.arange(T, dtype=torch.int32, device="cuda"), torch.zeros(T, H, dtype=x.dtype, device="cuda"),
                           most_rows=64)
        return out.split(counts)
    for a, b, n in zip(run(few), run(many), few):
        assert torch.equal(a, b[:n])
