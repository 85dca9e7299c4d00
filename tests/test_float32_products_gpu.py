"""32-bit products on the tensor cores: every form gives the same sums, and what is no number, very large or very small."""
import ctypes

import pytest
import torch

from test_float32_kernels_gpu import UNIT, k, rnd  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


def _form(k, x, w, cols, ranks):
    out = torch.full((x.shape[0] + 1, w.shape[0]), float("nan"), device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    status = k.lib.chibi_gemm_f32(p(x), p(w), p(out), None, x.shape[0], w.shape[0], x.shape[1], x.stride(0), w.stride(0), out.stride(0),
                                  0, cols, ranks, p(k.error), k._stream())
    assert status == 0
    k.check_error_word()
    assert torch.isnan(out[-1]).all()
    return out[:-1]


# K: less than a block, blocks that fill no run, one run to a half, runs cut short; N: less than a tile of 16 and of 128, more
# tiles of 16 than walkers
@pytest.mark.parametrize("N,K", [(5, 3), (130, 68), (40, 200), (300, 320), (129, 577), (5000, 1030), (64, 5000)])
def test_all_forms_give_the_same_sums(k, N, K):
    pad = -K % 4
    w, x = rnd(N, K + pad, seed=1)[:, :K], rnd(200, K + pad, seed=2)[:, :K]
    exact, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    whole = _form(k, x, w, 112, 1)
    # a block's sum: four roundings (the accumulator cuts off: twice as much) and the parts left out, below one; then the sums of
    # blocks, runs and halves
    blocks = -(-K // 64)
    assert ((whole.double() - exact).abs() <= (2 * 5 + 1 + blocks) * UNIT * size).all()
    for rows, cols in ((200, 128), (200, 16), (128, 128), (65, 80), (33, 48), (32, 32), (17, 32), (16, 16), (1, 16)):
        for ranks in (1, 2, 4, 8):
            assert torch.equal(_form(k, x[:rows], w, cols, ranks), whole[:rows]), (rows, cols, ranks)
    for rows in (1, 7, 8, 9, 16):
        for form in (4, 8, 16):
            assert torch.equal(_form(k, x[:rows], w, -form, 0), whole[:rows]), (rows, form)


@pytest.mark.parametrize("rows", [5, 12, 40, 150])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 3.4e38, 1e34])
def test_numbers_that_have_no_parts(k, rows, bad):
    N, K = 6000, 200
    x, w = rnd(rows, K, seed=3), rnd(N, K, seed=4)
    clean = torch.empty(rows, N, device="cuda")
    k.linear(x, w, clean)
    w[0, 1] = 0.0                                            # (an infinity times this is no number, whatever its parts are)
    x[3, 1] = x[0, 199] = bad
    w[50, 70] = w[5990, 70] = bad
    out = torch.empty(rows, N, device="cuda")
    k.linear(x, w, out)
    k.check_error_word()
    rest = torch.ones(rows, N, dtype=torch.bool, device="cuda")
    rest[[0, 3]] = False
    rest[:, [0, 50, 5990]] = False
    assert torch.equal(out[rest], clean[rest])
    exact = x.double() @ w.double().t()
    if bad < 3.5e38:
        small = exact.abs() < 3e38
        # (where both rows are marked, a sum on its way may pass the largest number although its end does not)
        small[[[0], [3]], [50, 5990]] = False
        bound = (K + 10) * UNIT * (x.double().abs() @ w.double().abs().t())
        assert ((out.double() - exact).abs() <= bound)[small].all() and torch.isinf(out[~small & (exact.abs() > 3.5e38)]).all()
    else:
        assert torch.equal(torch.isfinite(out), torch.isfinite(exact)) and torch.equal(torch.isnan(out), torch.isnan(exact))


@pytest.mark.parametrize("rows", [3, 40])
def test_small_activations_keep_their_bits(k, rows):
    x, w = rnd(rows, 256, seed=5) * 1e-37, rnd(70, 256, seed=6)
    out = torch.empty(rows, 70, device="cuda")
    k.linear(x, w, out)
    exact = x.double() @ w.double().t()
    # (beside the relative bound, half the spacing of numbers below 2^-126)
    assert ((out.double() - exact).abs() <= 15 * UNIT * (x.double().abs() @ w.double().abs().t()) + 2.0 ** -149).all()


def test_sums_too_large_for_scaled_accumulators(k):
    x, w = torch.full((20, 128), 2.0 ** 62, device="cuda"), torch.full((30, 128), 2.0 ** 57, device="cuda")
    for rows in (4, 20):                                     # 2^126; 2^16 as much is infinite
        out = torch.empty(rows, 30, device="cuda")
        k.linear(x[:rows], w, out)
        assert (out == 2.0 ** 126).all()


@pytest.mark.parametrize("x_size,w_size", [(1.0, 1e-35), (1.0, 1e-37), (1e30, 1e-37), (1e-20, 1e-17)])
@pytest.mark.parametrize("rows", [3, 12, 40])
def test_small_weights_keep_their_bits(k, rows, x_size, w_size):
    x, w = rnd(rows, 256, seed=5) * x_size, rnd(70, 256, seed=6) * w_size
    w[:, ::7] += 2.0 ** -126                                 # (the least normal number among them)
    out = torch.empty(rows, 70, device="cuda")
    k.linear(x, w, out)
    exact = x.double() @ w.double().t()
    # (as above; a number below 2^-126 has parts down to 2^-149, of which 2^-150 is lost at most)
    lost = 2.0 ** -149 + 2.0 ** -150 * x.double().abs().sum(1, keepdim=True)
    assert ((out.double() - exact).abs() <= 15 * UNIT * (x.double().abs() @ w.double().abs().t()) + lost).all()


# (one chain of roundings over K lost 5.8e-7 of the sizes here, 64-bit sums nothing: what is left is the result's rounding)
@pytest.mark.parametrize("rows", [4, 12, 40, 300])
def test_large_numbers_are_summed_exactly(k, rows):
    x, w, residual = rnd(rows, 1028, seed=9)[:, :1027], (rnd(300, 1028, seed=10) * 1e-3)[:, :1027], rnd(rows, 300, seed=11) * 1e33
    x[rows // 2] *= 1e35
    w[7] *= 1e37
    out = residual.clone()
    k.linear(x, w, out, out)                                 # (added in place)
    exact, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    large = torch.zeros(rows, 300, dtype=torch.bool, device="cuda")
    large[rows // 2] = large[:, 7] = True
    finite, total = exact.abs() < 3e38, exact + residual.double()
    assert ((out.double() - total).abs() <= 2 * UNIT * (exact.abs() + total.abs()))[large & finite].all()
    assert ((out.double() - total).abs() <= (15 + 17) * UNIT * size + 2 * UNIT * total.abs())[~large & finite].all()
    assert torch.isinf(out[exact.abs() > 3.5e38]).all()


# Operands of one sign: what the accumulators cut off does not cancel.  Of a block of 64 places four roundings, each of at most a
# unit of what is there (2 UNIT), the first three smaller; then the sums of blocks, runs and halves.  On average less: 2-norm
# 9.3e-8, 0.84e-7 of it one-sided, at every K; by multiply-adds 4.4e-8 to 9.2e-8.
@pytest.mark.parametrize("rows", [8, 12, 64])
@pytest.mark.parametrize("K", [64, 1024, 12288])
def test_operands_of_one_sign(k, rows, K):
    x, w = rnd(rows, K, seed=7).abs(), rnd(300, K, seed=8).abs()
    out = torch.empty(rows, 300, device="cuda")
    k.linear(x, w, out)
    exact = x.double() @ w.double().t()
    error = (out.double() - exact) / exact
    # (a sum of n blocks, each with its own error, has the average of theirs and the roundings of the sums in between)
    assert float(error.abs().max()) <= (2 * 5 + 1 + -(-K // 64)) * UNIT
    assert float(error.square().mean().sqrt()) <= 2 * UNIT and -2 * UNIT <= float(error.mean()) <= 0
