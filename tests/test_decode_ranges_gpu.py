"""Decode attention over sequences of different lengths: key ranges cut on the device by the sequences' lengths, and more
sequences than fit the SMs at once in the order of their lengths."""
import math

import pytest
import torch

from test_kernels_gpu import _paged_setup, close, k, ref, rnd  # noqa: F401 (fixtures)

pytestmark = pytest.mark.gpu


def _check(k, ref, lens, nq, nkv, d, window=None, page=16, q_lens=None, seed=0):
    q_lens = q_lens or [1] * len(lens)
    pages = sum(-(-n // page) for n in lens)
    table, positions, seq_of_token, q_start, ctx_len = _paged_setup(lens, q_lens, page, pages, seed=seed)
    q = rnd(sum(q_lens), nq * d, dtype=torch.bfloat16, seed=seed + 1)
    kc = rnd(pages, nkv, page, d, dtype=torch.bfloat16, seed=seed + 2)
    vc = rnd(pages, nkv, page, d, dtype=torch.bfloat16, seed=seed + 3)
    out = torch.full_like(q, float("nan"))
    exp = torch.empty_like(out)
    args = (table, q_start, ctx_len, seq_of_token, positions, nq, nkv, d, page, 1 / math.sqrt(d), window, max(q_lens),
            max(lens), min(q_lens))
    k.attention(q, kc, vc, out, *args)
    ref.attention(q, kc, vc, exp, *args)
    k.check_error_word()
    close(out, exp, torch.bfloat16, "decode attention", rel=1.2e-2)      # (as the other tests of this kernel)


@pytest.fixture
def always(k, monkeypatch):                   # (ranges by length for small contexts too)
    rule = type(k).decode_attention_units
    monkeypatch.setattr(type(k), "decode_attention_units", lambda self, seqs, nq, nkv, splits, longest: rule(
        self, seqs, nq, nkv, splits, max(longest, 512 * splits)))


# one long sequence among short ones; ranges at the least length; equal lengths; one sequence more than a warp's lanes
@pytest.mark.parametrize("lens", [[1, 3000], [2000] + [17] * 9, [129, 128, 127, 1, 640], [700] * 8,
                                  [5000, 16, 900, 33, 1200, 2500, 40], [300 + 61 * (i % 9) for i in range(33)]])
@pytest.mark.parametrize("nq,nkv,d", [(8, 4, 128), (4, 2, 64), (20, 1, 48), (3, 1, 16)])
def test_ranges_by_length(k, ref, always, lens, nq, nkv, d):
    splits = k.decode_attention_splits(len(lens), nq, nkv, max(lens))
    assert splits > 1 and k.decode_attention_units(len(lens), nq, nkv, splits, max(lens))[0] >= len(lens)
    _check(k, ref, lens, nq, nkv, d)


@pytest.mark.parametrize("window", [40, 500])
def test_ranges_by_length_in_a_window_beside_a_portion(k, ref, always, window):
    _check(k, ref, [3000, 700, 90, 1500, 260], 4, 2, 128, window=window, q_lens=[1, 1, 1, 37, 1])


@pytest.mark.parametrize("seqs", [127, 128, 129])
def test_the_most_sequences_that_are_cut_by_length(k, ref, always, seqs):
    lens = [1 + (197 * i) % 900 for i in range(seqs)]
    splits = k.decode_attention_splits(seqs, 2, 1, max(lens))
    assert splits > 1 and (k.decode_attention_units(seqs, 2, 1, splits, max(lens))[0] > 0) == (seqs <= 128)
    _check(k, ref, lens, 2, 1, 128)


@pytest.mark.parametrize("seqs,nkv,d", [(64, 8, 128), (127, 4, 64), (128, 8, 64), (129, 4, 64), (64, 8, 48)])
def test_longest_sequences_first(k, ref, seqs, nkv, d):
    lens = [1 + (331 * i) % 700 for i in range(seqs - 2)] + [1, 1024]      # (equal lengths among them)
    assert k.decode_attention_units(seqs, 2 * nkv, nkv, 1, 1024) == (0, int(seqs <= 128))
    assert k.decode_attention_splits(seqs, 2 * nkv, nkv, 1024) == 1
    _check(k, ref, lens, 2 * nkv, nkv, d)


# What follows attention in a model is a kernel that starts early and waits for the kernel ahead of it alone: for the merge,
# which in these steps has nothing to merge (a window or single tokens of at most 128 keys), or for a decode kernel without
# any single token (0: how many tokens a sequence brings at least is not said).
@pytest.mark.parametrize("lens,q_lens,window,least", [
    ([3000, 4096, 2100, 3500] * 2, [1] * 8, 40, 1), ([90, 40, 128, 1] * 4 + [1500], [1] * 16 + [200], None, 1),
    ([300, 500], [300, 100], None, 0)])
def test_the_product_behind_reads_finished_rows(k, ref, lens, q_lens, window, least):
    nq, nkv, d, page = 16, 8, 128, 16
    pages = sum(-(-n // page) for n in lens)
    table, positions, seq_of_token, q_start, ctx_len = _paged_setup(lens, q_lens, page, pages, seed=3)
    q = rnd(sum(q_lens), nq * d, dtype=torch.bfloat16, seed=4)
    kc = rnd(pages, nkv, page, d, dtype=torch.bfloat16, seed=5)
    vc = rnd(pages, nkv, page, d, dtype=torch.bfloat16, seed=6)
    w = rnd(256, nq * d, dtype=torch.bfloat16, seed=7, scale=0.02)
    args = (table, q_start, ctx_len, seq_of_token, positions, nq, nkv, d, page, 1 / math.sqrt(d), window, max(q_lens),
            max(lens), least)
    out, exp = torch.empty_like(q), torch.empty_like(q)
    product = torch.empty(q.shape[0], 256, dtype=torch.float32, device="cuda")
    ref.attention(q, kc, vc, exp, *args)
    expected = exp.float() @ w.float().t()

    def step():
        out.fill_(float("nan"))
        k.attention(q, kc, vc, out, *args)
        k.linear(out, w, product)

    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for run in [step] * 10 + [graph.replay] * 20:
        product.fill_(float("nan"))
        run()
        close(out, exp, torch.bfloat16, "attention", rel=1.2e-2)         # (as the other tests of this kernel)
        close(product, expected, torch.float32, "the product behind", rel=1.5e-2)    # (that of its rows, each 1.2e-2 at most)
    k.check_error_word()


def test_a_sequence_without_a_key_gives_zeros(k, always):
    nq, nkv, d, page, lens = 4, 2, 64, 16, [900, 0, 300, 40]
    splits = k.decode_attention_splits(len(lens), nq, nkv, max(lens))
    assert splits > 1 and k.decode_attention_units(len(lens), nq, nkv, splits, max(lens))[0] >= len(lens)
    pages = sum(-(-n // page) for n in lens)
    table, positions, seq_of_token, q_start, ctx_len = _paged_setup(lens, [1] * 4, page, pages, seed=1)
    q = rnd(4, nq * d, dtype=torch.bfloat16, seed=2)
    kc, vc = rnd(pages, nkv, page, d, dtype=torch.bfloat16, seed=3), rnd(pages, nkv, page, d, dtype=torch.bfloat16, seed=4)
    out = torch.full_like(q, float("nan"))
    k.attention(q, kc, vc, out, table, q_start, ctx_len, seq_of_token, positions, nq, nkv, d, page, d ** -0.5, None, 1, max(lens), 1)
    k.check_error_word()
    assert (out[1] == 0).all() and torch.isfinite(out).all()


@pytest.mark.parametrize("lens", [[2100, 2048, 2000, 1900] * 2, [5000, 16, 900, 33, 1200, 2500, 40], [4096] * 40, [4096, 100] * 20])
def test_a_hint_about_lengths_is_a_matter_of_time(k, ref, lens):
    nq, nkv, d, page = 16, 8, 128, 16
    pages = sum(-(-n // page) for n in lens)
    table, positions, seq_of_token, q_start, ctx_len = _paged_setup(lens, [1] * len(lens), page, pages, seed=1)
    q = rnd(len(lens), nq * d, dtype=torch.bfloat16, seed=2)
    kc, vc = rnd(pages, nkv, page, d, dtype=torch.bfloat16, seed=3), rnd(pages, nkv, page, d, dtype=torch.bfloat16, seed=4)
    args = (table, q_start, ctx_len, seq_of_token, positions, nq, nkv, d, page, 1 / math.sqrt(d), None, 1, max(lens), 1)
    exp = torch.empty_like(q)
    ref.attention(q, kc, vc, exp, *args)
    for even in (False, True):
        out = torch.full_like(q, float("nan"))
        k.attention(q, kc, vc, out, *args, even_contexts=even)
        k.check_error_word()
        close(out, exp, torch.bfloat16, "decode attention", rel=1.2e-2)      # (as the other tests of this kernel)
