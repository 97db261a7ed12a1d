"""The one-block dispatch (csrc/route.cu) at the edges of its slices and of its range: whole numbers, compared exactly with
a stable sort on the host; ids outside the table are clamped as everywhere."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 31, 33, 512, 1023, 1025, 2049, 4095, 4096, 4097])
@pytest.mark.parametrize("E", [1, 7, 33, 64, 256])
def test_dispatch(T, E):
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(T * 300 + E)
    V = 1000
    table = torch.randint(0, E, (V,), generator=g)
    if E > 3:
        table[table == 2] = 3                                # an expert without tokens
    ids = torch.randint(-5, V + 5, (T,), generator=g)
    r = ops.route(ids.cuda(), table.cuda(), E)
    want = table[ids.clamp(0, V - 1)]
    perm = torch.sort(want, stable=True).indices
    assert torch.equal(r.expert_ids.cpu().long(), want) and torch.equal(r.perm.cpu().long(), perm)
    assert torch.equal(r.inv_perm.cpu().long()[perm], torch.arange(T))
    counts = torch.bincount(want, minlength=E)
    assert torch.equal(r.counts.cpu().long(), counts)
    assert torch.equal(r.offsets.cpu().long(), torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]))
