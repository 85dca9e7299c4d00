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


def exact_attention(q, keys, values, table, q_lens, ctx, nq, nkv, d, page, scale, window, chunk, softcap, bias, sink):
    out, at, G = [], 0, nq // nkv
    for s, (n, c) in enumerate(zip(q_lens, ctx)):
        pages = table[s, :-(-c // page)].long().clamp(min=0)
        k = keys[pages].transpose(1, 2).reshape(-1, nkv, d)[:c].double().repeat_interleave(G, 1)
        v = values[pages].transpose(1, 2).reshape(-1, nkv, d)[:c].double().repeat_interleave(G, 1)
        x = torch.einsum("thd,khd->htk", q[at:at + n].view(n, nq, d).double(), k) * scale
        if softcap:
            x = softcap * torch.tanh(x / softcap)
        i, j = torch.arange(c - n, c, device="cuda")[:, None], torch.arange(c, device="cuda")[None]
        if bias is not None:
            r1, r2 = (None if r is None else r.double()[:, None, None] for r in bias)
            x = x - (r1 * (i - j).double() if r2 is None else r1 * torch.log1p(r2 * (i - j).clamp(min=0).double()))
        hidden = j > i
        if window:
            hidden = hidden | (j <= i - window)
        if chunk:
            hidden = hidden | (j < i - i % chunk)
        x = x.masked_fill(hidden, float("-inf"))
        if sink is not None:
            x = torch.cat([x, sink.double()[:, None, None].expand(nq, n, 1)], -1)
            v = torch.cat([v, torch.zeros_like(v[:1])])
        out.append(torch.einsum("htk,khd->thd", torch.softmax(x, -1), v).reshape(n, nq * d))
        at += n
    return torch.cat(out)


# lengths: single tokens with 1 key, a range's edge (64 keys), eight ranges and more; portions that begin inside a tile
# of 32 keys; row tiles cut inside a token's group (5 heads) and by the sequence's end; steps of both kinds
@pytest.mark.parametrize("d,nq,nkv,page,q_lens,ctx,options", [
    (128, 4, 2, 16, [1, 1, 1, 1], [1, 64, 65, 1500], {}),
    (64, 5, 1, 8, [1, 1, 1], [33, 512, 513], {"softcap": 20.0, "sink": True}),
    (64, 16, 2, 16, [1, 1], [300, 700], {"window": 100, "bias": "linear"}),
    (64, 4, 4, 32, [1, 1], [300, 40], {"chunk": 64, "bias": "log"}),
    (128, 4, 2, 16, [2, 33, 130], [2, 40, 330], {}),
    (64, 5, 1, 8, [100, 13], [100, 77], {"softcap": 20.0, "sink": True}),
    (64, 16, 2, 16, [70, 1, 5], [300, 90, 5], {"window": 50, "bias": "linear"}),
    (128, 4, 4, 32, [150, 1], [200, 1], {"chunk": 64, "bias": "log"}),
])
def test_attention_float32(k, d, nq, nkv, page, q_lens, ctx, options):
    T, S = sum(q_lens), len(q_lens)
    pages = [-(-c // page) for c in ctx]
    order = torch.randperm(sum(pages) + 3, generator=torch.Generator().manual_seed(1)).to(torch.int32)
    table = torch.zeros(S, max(pages) + 1, dtype=torch.int32)
    at = 0
    for s, n in enumerate(pages):
        table[s, :n] = order[at:at + n]
        at += n
    # pages that every query's window or block has left behind are gone
    for s, (n, c) in enumerate(zip(q_lens, ctx)):
        i = c - n
        oldest = max(i - options["window"] + 1 if options.get("window") else 0,
                     i - i % options["chunk"] if options.get("chunk") else 0, 0)
        table[s, :oldest // page] = -1
    table = table.cuda()
    keys, values = rnd(sum(pages) + 3, nkv, page, d, seed=1), rnd(sum(pages) + 3, nkv, page, d, seed=2)
    q = rnd(T, nq * d, seed=3)
    # what nobody may read: places past a sequence's end in its last page, and pages of nobody
    used = torch.zeros(keys.shape[0], page, dtype=torch.bool, device="cuda")
    for s, c in enumerate(ctx):
        for u in range(c):
            if table[s, u // page] >= 0:
                used[table[s, u // page].long(), u % page] = True
    keys.masked_fill_(~used[:, None, :, None], float("nan"))
    values.masked_fill_(~used[:, None, :, None], float("nan"))
    starts = [0]
    for n in q_lens:
        starts.append(starts[-1] + n)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    bias = {None: None, "linear": (rnd(nq, seed=4).abs() * 0.1, None),
            "log": (rnd(nq, seed=4).abs(), rnd(nq, seed=5).abs())}[options.get("bias")]
    sink = rnd(nq, seed=6) if options.get("sink") else None
    out = torch.full((T, nq * d), float("nan"), device="cuda")
    k.attention(q, keys, values, out, table, ints(starts), ints(ctx), ints([i for i, n in enumerate(q_lens) for _ in range(n)]),
                ints([c - n + j for n, c in zip(q_lens, ctx) for j in range(n)]), nq, nkv, d, page, d ** -0.5,
                options.get("window"), max(q_lens), max(ctx), min_q_len=min(q_lens), softcap=options.get("softcap"),
                distance_bias=bias, chunk=options.get("chunk"), sink=sink)
    k.check_error_word()
    exact = exact_attention(q, keys.nan_to_num(), values.nan_to_num(), table, q_lens, ctx, nq, nkv, d, page, d ** -0.5,
                            options.get("window"), options.get("chunk"), options.get("softcap"), bias, sink)
    # a score is off by at most (d / 4 + 8) roundings of sums of magnitude |q| |k| / sqrt(d) < 16, its exponential by
    # as much relatively, and the weighted mean of values below 6 by twice that
    assert torch.isfinite(out).all()
    assert float((out.double() - exact).abs().max()) <= 2 * 6 * 16 * (d / 4 + 16) * UNIT


def test_attention_float32_hides_later_values(k):
    """A value that is not a number reaches only the tokens that see its key."""
    d, T = 64, 40
    keys, values, q = rnd(3, 1, 16, d, seed=1), rnd(3, 1, 16, d, seed=2), rnd(T, d, seed=3)
    values[1, 0, 4] = float("nan")                       # position 20
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    out = torch.empty(T, d, device="cuda")
    k.attention(q, keys, values, out, ints([[0, 1, 2]]), ints([0, T]), ints([T]), ints([0] * T), ints(list(range(T))), 1, 1, d, 16,
                d ** -0.5, None, T, T, min_q_len=T)
    assert torch.isfinite(out[:20]).all() and torch.isnan(out[20:]).all()


@pytest.mark.parametrize("ranks", [1, 2, 4])
def test_single_tokens_with_fewer_ranges_than_keys(k, ranks, monkeypatch):
    """A step captured while contexts were short runs on: its CTAs then take several ranges each."""
    d, c = 64, 900
    keys, values, q = rnd(60, 2, 16, d, seed=1), rnd(60, 2, 16, d, seed=2), rnd(1, 4 * d, seed=3)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    table, out = ints([list(range(57))]), torch.full((1, 4 * d), float("nan"), device="cuda")
    monkeypatch.setattr(type(k), "float32_token_ranks", staticmethod(lambda n: ranks))
    k.attention(q, keys, values, out, table, ints([0, 1]), ints([c]), ints([0]), ints([c - 1]), 4, 2, d, 16, d ** -0.5, None, 1, c,
                min_q_len=1)
    exact = exact_attention(q, keys, values, table, [1], [c], 4, 2, d, 16, d ** -0.5, None, None, None, None, None)
    assert float((out.double() - exact).abs().max()) <= 2 * 6 * 16 * (d / 4 + 16) * UNIT


@pytest.mark.parametrize("rows", [1, 2, 4, 8, 16, 48, 70, 300])
def test_linear_float32_reads_weights_that_the_kernel_ahead_wrote(k, rows):
    """Every kernel starts before the one ahead has ended: no weight is read before that."""
    N, K = 4096, 1024
    first, x = rnd(N, K, seed=7), rnd(rows, K, seed=8)
    for wait in (True, False, False, False):
        ws, outs = [first.clone() for _ in range(4)], [torch.full((rows, N), float("nan"), device="cuda") for _ in range(4)]
        torch.cuda.synchronize()
        for w, out in zip(ws, outs):
            k.scale(w, 2.0)
            if wait:
                torch.cuda.synchronize()
            k.linear(x, w, out)
        torch.cuda.synchronize()
        if wait:
            right = outs
        assert all(torch.equal(a, b) for a, b in zip(outs, right))
    plain = torch.full((rows, N), float("nan"), device="cuda")
    k.linear(x, first, plain)                            # (a power of two scales every sum exactly)
    assert torch.equal(right[0], 2 * plain)
