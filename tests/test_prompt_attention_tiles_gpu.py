"""Prompt attention on tcgen05 at the edges of its query tiles: whole tokens of a group's heads to a tile (queries by TMA) or
not (gathered), with one and with two tiles to a CTA."""
import math

import pytest
import torch

from test_kernels_gpu import _paged_setup, close, k, ref, rnd  # noqa: F401 (fixtures)

pytestmark = pytest.mark.gpu


# rows of a tile: one token more or less than a tile, than two tiles, than a tile of keys; a tile of one token
@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("nq,nkv,d,lens", [(8, 2, 128, [65, 31, 129]), (4, 4, 64, [128, 257, 127]), (10, 2, 128, [26, 52, 103]),
                                           (6, 2, 64, [43, 86]), (128, 1, 64, [2, 5]), (16, 2, 128, [16, 33, 130])])
@pytest.mark.parametrize("options", [{}, {"softcap": 20.0}, {"window": 40}])
def test_query_tiles(k, ref, monkeypatch, variant, nq, nkv, d, lens, options):
    monkeypatch.setattr(k, "tcgen05_attention_variant", variant)
    ctx = [n + 37 * (i % 2) for i, n in enumerate(lens)]
    page, pages = 16, sum(-(-c // 16) for c in ctx)
    table, positions, seq_of_token, q_start, ctx_len = _paged_setup(ctx, lens, page, pages, seed=1)
    q = rnd(sum(lens), nq * d, dtype=torch.bfloat16, seed=2)
    kc, vc = rnd(pages, nkv, page, d, dtype=torch.bfloat16, seed=3), rnd(pages, nkv, page, d, dtype=torch.bfloat16, seed=4)
    exp = torch.empty_like(q)
    args = (table, q_start, ctx_len, seq_of_token, positions, nq, nkv, d, page, 1 / math.sqrt(d), options.get("window"), max(lens),
            max(ctx))
    more = dict(min_q_len=min(lens), softcap=options.get("softcap"))
    ref.attention(q, kc, vc, exp, *args, **more)
    # the next sequence's first token is no number: a tile that reaches into it must not show that
    first = int(q_start[1])
    q[first] = float("nan")
    out = torch.full((q.shape[0] + 1, nq * d), 7.0, dtype=torch.bfloat16, device="cuda")
    k.attention(q, kc, vc, out[:-1], *args, **more)
    k.check_error_word()
    assert torch.isnan(out[first]).all() and (out[-1] == 7.0).all()
    rest = [i for i in range(q.shape[0]) if i != first]
    close(out[rest], exp[rest], torch.bfloat16, "prompt attention", rel=1.2e-2)        # (as the other tests of these kernels)
