"""The kernels of the 32-bit path against 64-bit arithmetic, at the edges of their tiles and parts."""
import pytest
import torch

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -24


@pytest.fixture(scope="module")
def k():
    from chibillm_b200.kernels.ops import CudaKernels
    return CudaKernels(torch.device("cuda:0"))


def rnd(*shape, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda")


# rows: each width of the few-row kernel and its padding, blocks of 16, the tiles' height and remainders; N: a lone
# column, remainders of 32 and 64, tiles shared by 1, 2 and 4 CTAs, more tiles than CTAs, two rows a lane; K: less than
# a block, no whole block, one part, a last part that is cut short, sixteen parts
@pytest.mark.parametrize("N,K", [(1, 4), (70, 36), (96, 100), (1024, 1024), (1000, 3072), (4224, 2052), (9700, 132), (64, 12300)])
def test_linear_float32(k, N, K):
    w, x_all, residual = rnd(N, K, seed=1), rnd(300, K + 4, seed=2)[:, :K], rnd(300, N, seed=3)
    exact = x_all.double() @ w.double().t()
    # a part of max(K / 16, 128) places (rounded up to 32) and 16 parts: so many roundings of partial sums, each of at
    # most the sum of the magnitudes
    bound = (max(K / 16, 128) + 60) * UNIT * (x_all.double().abs() @ w.double().abs().t()) + 4 * UNIT * residual.double().abs()
    whole = torch.full((300, N), float("nan"), device="cuda")
    k.linear(x_all, w, whole)
    assert ((whole.double() - exact).abs() <= bound).all()
    for rows in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 48, 49, 64, 65):
        out = torch.full((rows + 1, N), float("nan"), device="cuda")
        k.linear(x_all[:rows], w, out[:rows])
        assert torch.equal(out[:rows], whole[:rows]), f"{rows} rows: not the sums of 300 rows"
        assert torch.isnan(out[rows]).all()
        acc = residual[:rows].clone()
        k.linear(x_all[:rows], w, acc, residual=acc)
        assert ((acc.double() - exact[:rows] - residual[:rows].double()).abs() <= bound[:rows]).all()


def test_linear_float32_keeps_infinities_to_their_rows(k):
    x, w = rnd(70, 200, seed=4), rnd(100, 200, seed=5)
    x[3, 7], w[50, 199] = float("inf"), float("nan")
    for rows in (8, 20, 70):
        out = torch.empty(rows, 100, device="cuda")
        k.linear(x[:rows], w, out)
        bad = ~torch.isfinite(out)
        assert bad[3].all() and bad[:, 50].all() and int(bad.sum()) == 100 + rows - 1
