"""The activation of a gated feed-forward, four values a thread and one."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("tx,to", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32),
                                   (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("rows,inter", [(1, 4), (3, 6), (4, 252), (5, 260), (127, 1020), (128, 1028), (129, 44), (65536, 4)])
def test_swiglu(tx, to, rows, inter):
    from chibillm_b200.kernels.ops import CudaKernels
    k = CudaKernels(torch.device(DEV))
    g = torch.Generator(device=DEV).manual_seed(rows)
    x = (torch.randn(rows, 2 * inter, generator=g, device=DEV) * 5).to(tx)
    x[0, 0], x[-1, -1] = 100.0, -1.0
    out = torch.full((rows, inter), float("nan"), device=DEV, dtype=to)
    k.swiglu(x, out)
    gate, up = x.double().split(inter, 1)
    ref = gate * torch.sigmoid(gate) * up
    # the exponential (two units of 2^-23, and its argument is exact), a sum, a division and a product (half a unit each), the
    # rounding of the result: half a unit of its 8th or 24th significant bit
    last = 2.0 ** -8 if to == torch.bfloat16 else 2.0 ** -24
    assert ((out.double() - ref).abs() <= (5 * 2.0 ** -23 + last * 1.01) * ref.abs() + 1e-37).all()
