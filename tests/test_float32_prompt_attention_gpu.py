"""32-bit prompt attention: a row's result against 64-bit arithmetic and beside other rows, and numbers that are none."""
import pytest
import torch

from test_float32_kernels_gpu import UNIT, exact_attention, k, rnd  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


def _ints(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _run(k, q, keys, values, table, q_lens, ctx, nq, nkv, d, page, **more):
    starts = [0]
    for n in q_lens:
        starts.append(starts[-1] + n)
    out = torch.full((q.shape[0] + 1, nq * d), 7.0, device="cuda")
    k.attention(q, keys, values, out[:-1], table, _ints(starts), _ints(ctx), _ints([i for i, n in enumerate(q_lens) for _ in range(n)]),
                _ints([c - n + j for n, c in zip(q_lens, ctx) for j in range(n)]), nq, nkv, d, page, d ** -0.5, more.get("window"),
                max(q_lens), max(ctx), min_q_len=min(q_lens))
    k.check_error_word()
    assert (out[-1] == 7.0).all()
    return out[:-1]


# tiles of 128 rows and blocks of 64 keys: one more and one less of each, a tile cut inside a token's heads, a tile of one token
@pytest.mark.parametrize("d,nq,nkv,page,q_lens,ctx,window", [
    (128, 2, 1, 16, [64, 65, 63], [64, 65, 63], None), (64, 4, 4, 8, [128, 129, 2], [128, 129, 130], None),
    (128, 3, 1, 32, [43, 44], [191, 193], 70), (64, 130, 1, 16, [2, 3], [2, 67], None), (64, 2, 2, 1, [130], [513], 64)])
def test_tiles(k, d, nq, nkv, page, q_lens, ctx, window):
    pages = [-(-c // page) for c in ctx]
    table = torch.zeros(len(ctx), max(pages), dtype=torch.int32)
    at = 0
    for s, n in enumerate(pages):
        table[s, :n] = torch.arange(at, at + n)
        at += n
    table = table.cuda()
    keys, values, q = rnd(at, nkv, page, d, seed=1), rnd(at, nkv, page, d, seed=2), rnd(sum(q_lens), nq * d, seed=3)
    out = _run(k, q, keys, values, table, q_lens, ctx, nq, nkv, d, page, window=window)
    exact = exact_attention(q, keys, values, table, q_lens, ctx, nq, nkv, d, page, d ** -0.5, window, None, None, None, None)
    # (the bound of test_attention_float32: what the scores, |q| |k| / sqrt(d) < 16, the exponentials and the mean lose)
    assert float((out.double() - exact).abs().max()) <= 2 * 6 * 16 * (d / 4 + 16) * UNIT


@pytest.mark.parametrize("d", [64, 128])
def test_a_row_is_the_same_in_every_portion(k, d):
    nq, nkv, page, T = 4, 2, 16, 300
    keys, values, q = rnd(19, nkv, page, d, seed=4), rnd(19, nkv, page, d, seed=5), rnd(T, nq * d, seed=6)
    table = torch.arange(19, dtype=torch.int32, device="cuda")[None]
    whole = _run(k, q, keys, values, table, [T], [T], nq, nkv, d, page)
    at = 0
    for n in (2, 31, 100, 67, 100):
        assert torch.equal(_run(k, q[at:at + n], keys, values, table, [n], [at + n], nq, nkv, d, page), whole[at:at + n])
        at += n


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_numbers_that_are_none_stay_with_the_rows_that_see_them(k, d, bad):
    T, page = 200, 16
    q = rnd(T, d, seed=1)
    table = torch.arange(13, dtype=torch.int32, device="cuda")[None]
    clean = _run(k, q, rnd(13, 1, page, d, seed=2), rnd(13, 1, page, d, seed=3), table, [T], [T], 1, 1, d, page)
    near = lambda a, b: float((a - b).abs().max()) <= 2 * 6 * 16 * (d / 4 + 16) * UNIT
    for place in (70, 131):
        keys, values = rnd(13, 1, page, d, seed=2), rnd(13, 1, page, d, seed=3)
        values[place // page, 0, place % page, 5] = bad
        out = _run(k, q, keys, values, table, [T], [T], 1, 1, d, page)
        assert torch.equal(out[:place], clean[:place])
        others = [c for c in range(d) if c != 5]
        assert not torch.isfinite(out[place:, 5]).any() and near(out[place:, others], clean[place:, others])
        keys, values = rnd(13, 1, page, d, seed=2), rnd(13, 1, page, d, seed=3)
        keys[place // page, 0, place % page, 7] = bad
        out = _run(k, q, keys, values, table, [T], [T], 1, 1, d, page)
        # an infinite key's score is an infinity of the query's sign: the lowest weighs nothing, the highest leaves no number
        lost = torch.full((T - place,), True, device="cuda") if bad != bad else q[place:, 7] * bad > 0
        assert torch.equal(out[:place], clean[:place])
        assert torch.isnan(out[place:][lost]).all() and torch.isfinite(out[place:][~lost]).all()
        asked = q.clone()
        asked[place, 3] = bad
        keys[place // page, 0, place % page, 7] = 0.5
        values = rnd(13, 1, page, d, seed=3)
        out = _run(k, asked, rnd(13, 1, page, d, seed=2), values, table, [T], [T], 1, 1, d, page)
        rest = [t for t in range(T) if t != place]
        assert torch.equal(out[rest], clean[rest]) and not torch.isfinite(out[place]).all()


@pytest.mark.parametrize("d", [64, 128])
def test_values_beyond_the_largest_bfloat16(k, d):
    T = 66
    q, keys, values = rnd(T, d, seed=1), rnd(5, 1, 16, d, seed=2), rnd(5, 1, 16, d, seed=3)
    values[0, 0, 0, 1] = 3.4e38                              # (rounded to bfloat16 it would be infinite)
    table = torch.arange(5, dtype=torch.int32, device="cuda")[None]
    out = _run(k, q, keys, values, table, [T], [T], 1, 1, d, 16)
    exact = exact_attention(q, keys, values, table, [T], [T], 1, 1, d, 16, d ** -0.5, None, None, None, None, None)
    assert torch.isfinite(out).all()
    assert float(((out.double() - exact)[:, 1] / exact[:, 1]).abs().max()) <= 2 * 16 * (d / 4 + 16) * UNIT


# small and large numbers: last parts down to the least normal number; products, sums of scores and sums of values that a scaled
# accumulator cannot hold
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("q_size,k_size,v_size", [(1.0, 1.0, 1e-36), (1.0, 1.0, 1e-37), (1e-36, 1e36, 1.0), (1e35, 1e-35, 1.0),
                                                  (1e-20, 1e20, 1e33), (1.0, 1.0, 1e37)])
def test_small_and_large_numbers(k, d, q_size, k_size, v_size):
    nq, nkv, page, q_lens, ctx = 4, 2, 16, [140, 2, 66], [140, 300, 66]
    pages = [-(-c // page) for c in ctx]
    table = torch.zeros(3, max(pages), dtype=torch.int32)
    for s, n in enumerate(pages):
        table[s, :n] = torch.arange(sum(pages[:s]), sum(pages[:s]) + n)
    table = table.cuda()
    keys, values = rnd(sum(pages), nkv, page, d, seed=1) * k_size, rnd(sum(pages), nkv, page, d, seed=2) * v_size
    q = rnd(sum(q_lens), nq * d, seed=3) * q_size
    out = _run(k, q, keys, values, table, q_lens, ctx, nq, nkv, d, page)
    exact = exact_attention(q, keys, values, table, q_lens, ctx, nq, nkv, d, page, d ** -0.5, None, None, None, None, None)
    # (the bound of test_tiles, times the values' size; a value below 2^-126 loses 2^-150 at most)
    assert float((out.double() - exact).abs().max()) <= 2 * 6 * 16 * (d / 4 + 16) * UNIT * v_size + 2.0 ** -148
    # (and no more than multiply-adds, which lost 1.8e-7 and 2.2e-7 of these numbers at every size)
    relative = float((out.double() - exact).norm() / exact.norm())
    assert relative <= 2.5e-7, relative


@pytest.mark.parametrize("d", [64, 128])
def test_a_large_value_stays_with_the_rows_that_see_it(k, d):
    T, page, place = 200, 16, 131
    q, keys, values = rnd(T, d, seed=1), rnd(13, 1, page, d, seed=2), rnd(13, 1, page, d, seed=3)
    table = torch.arange(13, dtype=torch.int32, device="cuda")[None]
    clean = _run(k, q, keys, values, table, [T], [T], 1, 1, d, page)
    values[place // page, 0, place % page, 5] = 1e38
    values[place // page, 0, place % page, 6] = float("inf")
    out = _run(k, q, keys, values, table, [T], [T], 1, 1, d, page)
    exact = exact_attention(q, keys, values, table, [T], [T], 1, 1, d, page, d ** -0.5, None, None, None, None, None)
    assert torch.equal(out[:place], clean[:place]) and (out[place:, 6] == float("inf")).all()
    others = [c for c in range(d) if c not in (5, 6)]
    assert float((out.double() - exact)[place:, others].abs().max()) <= 2 * 6 * 16 * (d / 4 + 16) * UNIT
    assert float(((out.double() - exact)[place:, 5] / exact[place:, 5]).abs().max()) <= 2 * 16 * (d / 4 + 16) * UNIT
