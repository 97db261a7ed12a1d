"""Row groups that stream their weights with more than 64 rows in all (csrc/gemm_few_rows.cu): up to 8 a group on average
where the caller says that no group has more than 64. The kernel itself takes any number (most rows in one group among
them); only the choice goes by what was said."""
import pytest
import torch

import test_gpu_n_few_rows as few

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,H,I,bn,shared", [
    ([1] * 63 + [65], 72, 40, 64, 0), ([16] * 12, 264, 72, 256, 40), ([0] * 15 + [256], 104, 48, 128, 0), ([17] * 9, 64, 24, 32, 0),
    ([33, 0, 31] + [0] * 5, 520, 136, 256, 0), ([8] * 64, 40, 200, 256, 0), ([9] + [8] * 15, 72, 40, 64, 0), ([0] * 19 + [100, 60], 104, 48, 32, 0)])
def test_row_groups(counts, H, I, bn, shared):
    few.check_row_groups(counts, H, I, bn, shared, 64)


@pytest.mark.parametrize("counts", [[128] + [0] * 15, [64, 1] + [0] * 6 + [63] + [0] * 7])
def test_long_groups_stream_only_where_they_are_known_to_be_short(counts):
    """With no bound on a group, or one above 64 rows, a call of more than 64 rows has the bits of the tile kernel (which
    takes any call with more than 8 rows a group, here one row more); with a bound those of its first 64 rows streamed by
    themselves."""
    from complexity_deep_b200 import ops
    T, E, H, I, bn = 128, len(counts), 1032, 200, 64
    g = torch.Generator().manual_seed(T)
    seg = torch.tensor([0] + counts).cumsum(0).int().cuda()
    x, gate, up = (few._rand(g, *s, scale=0.1).cuda() for s in ((T + 1, H), (E, I, H), (E, I, H)))
    packed = ops.pack_gate_up(gate, up, bn)
    down, h = (few._rand(g, *s, scale=0.1).cuda() for s in ((E, H, I), (T + 1, I)))
    longer, short = seg.clone(), seg.clamp(max=64)
    longer[-1] += 1
    calls = [(lambda n, s, m: ops.glu_up(x[:n], packed, I, bn, 1.7, 7.0, 1.0, seg_offsets=s, most_rows=m)),
             (lambda n, s, m: ops.moe_down(h[:n], down, None, None, s, E, None, None, most_rows=m))]
    for call in calls:
        tiles, streamed = call(T + 1, longer, 64)[:T], call(64, short, 0)
        for most in (0, 65, T):
            assert torch.equal(call(T, seg, most), tiles), most
        assert not torch.equal(streamed, tiles[:64])
        assert torch.equal(call(T, seg, 64)[:64], streamed)
    up_only = ops.moe_up(x[:T], seg, E, packed, I, bn)
    assert torch.equal(up_only, ops.moe_up(x, longer, E, packed, I, bn)[:T])
    ops.status_fetch()
