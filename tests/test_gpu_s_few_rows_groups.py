"""Row groups that stream their weights with more than 64 rows in all (csrc/gemm_few_rows.cu): up to 8 a group on average,
most of them in one group among them, at the last call that streams and the first that does not."""
import pytest

import test_gpu_n_few_rows as few

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,H,I,bn,shared", [
    ([1] * 63 + [65], 72, 40, 64, 0), ([16] * 12, 264, 72, 256, 40), ([0] * 15 + [256], 104, 48, 128, 0), ([17] * 9, 64, 24, 32, 0),
    ([33, 0, 31] + [0] * 5, 520, 136, 256, 0), ([8] * 64, 40, 200, 256, 0), ([9] + [8] * 15, 72, 40, 64, 0), ([0] * 19 + [100, 60], 104, 48, 32, 0)])
def test_row_groups(counts, H, I, bn, shared):
    few.test_row_groups(counts, H, I, bn, shared)
