"""Sum of the chosen rows into the stream and the gather of rows (csrc/routed_experts.cu): more and fewer choices than are
loaded at a time, widths around a block's columns, more choices than a block notes at once; in the order of the choices,
so that 32-bit rows agree with the same chain of fused multiply-adds in 64 bits to `top` roundings."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("T,top,ldx", [(1, 1, 8), (3, 5, 1016), (64, 8, 2048), (7, 4, 1032), (2, 129, 2056), (300, 3, 600)])
def test_combine_and_gather(T, top, ldx, dtype):
    from complexity_deep_b200 import ops
    g = torch.Generator().manual_seed(T * top)
    y, w, x = torch.randn(T * top, ldx, generator=g).to(dtype), torch.rand(T, top, generator=g), torch.randn(T, ldx, generator=g)
    inv = torch.randperm(T * top, generator=g).int()
    rows = y.double()[inv.long()].view(T, top, ldx) * w.double()[..., None]
    want = x.double() + 0.5 * rows.sum(1)
    got = ops.combine_top_(x.cuda(), y.cuda(), inv.cuda(), w.cuda(), 0.5).double().cpu()
    assert bool(((got - want).abs() <= (top + 3) * 2.0 ** -24 * (rows.abs().sum(1) + x.double().abs())).all())
    assert torch.equal(ops.gather_div(x.to(dtype).cuda(), inv.cuda(), top).cpu(), x.to(dtype)[(inv.long() // top)])
