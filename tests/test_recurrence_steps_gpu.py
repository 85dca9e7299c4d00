"""Steps of few tokens of many sequences: the recurrences' kernels for full servers against the ones for few sequences."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def k():
    from chibillm_b200.kernels.ops import CudaKernels
    return CudaKernels(torch.device(DEV))


def ints(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


# heads x columns of 32 x sequences reach four warps an SM (592) in one call and stay below it sequence by sequence; key
# rows and value columns that fill no whole 32, 64 or 128
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,d,e", [(4, 20, 40), (4, 64, 64), (6, 50, 33), (3, 128, 72), (4, 100, 128)])
@pytest.mark.parametrize("rule", ["delta", "decayed"])
def test_many_sequences_equal_single_ones(k, rule, dtype, heads, d, e):
    g = torch.Generator(device=DEV).manual_seed(d)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    seqs = 100
    lens = [1 + (i * 7) % 4 for i in range(seqs)]
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    T = starts[-1]
    qkv = rnd(T, heads * (2 * d + e)).to(dtype)
    logits, beta, a_log, bias = rnd(T, heads * d), rnd(T, heads).to(dtype), rnd(heads), rnd(heads * d)
    decay = torch.rand(heads, generator=g, device=DEV)
    first = rnd(seqs + 1, heads, d, e)

    def run(state, o, a, b, slots, longest):
        q_start = ints([s - starts[a] for s in starts[a:b + 1]])
        rows = slice(starts[a], starts[b])
        if rule == "delta":
            k.channel_delta(qkv[rows], logits[rows], beta[rows], a_log, bias, state, o[rows], q_start, ints(slots), heads, heads,
                            d, e, 1e-6, d ** -0.5, longest)
        else:
            k.decayed_attention(qkv[rows], decay, state, o[rows], q_start, ints(slots), heads, d, e, longest, activate=True)

    assert heads * -(-e // 32) * seqs >= 592 > heads * -(-e // 32)
    slots = [(i * 37) % seqs for i in range(seqs)]
    one, many = first.clone(), first.clone()
    o1, o2 = torch.full((T, heads * e), float("nan"), device=DEV), torch.full((T, heads * e), float("nan"), device=DEV)
    run(many, o2, 0, seqs, slots, 4)
    for i in range(seqs):
        run(one, o1, i, i + 1, slots[i:i + 1], lens[i])
    # the same multiply-adds with the sums over the d rows in another order: d / 2 roundings of sums of magnitude
    # sqrt(d) max|S| at most (unit keys and queries of the delta rule; plain ones of the other)
    scale = float(o1.abs().max())
    assert float((o1 - o2).abs().max()) <= (d / 2 + 16) * 2.0 ** -24 * 4 * scale
    assert float((one - many).abs().max()) <= (d / 2 + 16) * 2.0 ** -24 * 4 * float(one.abs().max())
    assert torch.equal(many[seqs], first[seqs])


# heads: whole columns to a lane from 592 warps on, rows over warps below; d 200 has rows beyond 128
@pytest.mark.parametrize("seqs,d", [(1, 64), (1, 128), (1, 200), (8, 64), (8, 128), (8, 200), (200, 64)])
@pytest.mark.parametrize("rule", ["delta", "decayed", "general", "state space"])
def test_steps_without_a_wait_between_them_go_on_from_each_other(k, rule, seqs, d):
    """Each call finds the state that the one before it left, though the kernels start before that one has ended."""
    heads, steps = 2, 24
    g = torch.Generator(device=DEV).manual_seed(seqs + d)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x, logits, beta = rnd(steps, seqs, 5 * heads * d + 8), rnd(steps, seqs, heads * d), rnd(steps, seqs, heads)
    a_log, bias, removal = rnd(heads), rnd(heads * d), rnd(heads * d)
    decay = torch.rand(heads, generator=g, device=DEV)
    starts, slots = ints(list(range(seqs + 1))), ints(list(range(seqs)))
    first = rnd(seqs, heads, d, d)

    def run(wait):
        state, out = first.clone(), torch.full((steps, seqs, heads * d), float("nan"), device=DEV)
        torch.cuda.synchronize()
        for t in range(steps):
            if rule == "delta":
                k.channel_delta(x[t][:, :3 * heads * d], logits[t], beta[t], a_log, bias, state, out[t], starts, slots, heads,
                                heads, d, d, 1e-6, d ** -0.5, 1)
            elif rule == "decayed":
                k.decayed_attention(x[t][:, :3 * heads * d], decay, state, out[t], starts, slots, heads, d, d, 1)
            elif rule == "general":
                k.delta_rule(x[t], logits[t], bias, removal, state, out[t], starts, slots, heads, d, 8, 0.6, 1e-6, 1)
            else:
                k.state_space_scan(x[t][:, :3 * heads * d], beta[t], a_log, a_log, a_log, state, out[t], starts, slots, heads,
                                   heads, d, d)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return state, out

    state, out = run(True)
    assert torch.isfinite(out).all()
    for _ in range(3):
        again = run(False)
        assert torch.equal(again[0], state) and torch.equal(again[1], out)


# lengths: single tokens only (the kernel for few tokens), single tokens beside a prompt's portion (each kernel its own, the
# scan's at the edges of four tokens and of its chunks of 16), more than four tokens a sequence on average (the scan)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens,launches", [([1] * 20, 1), ([1, 4, 1], 1), ([1] * 63 + [190], 2), ([1, 5, 4, 1], 2), ([3, 16, 1, 1, 1, 2], 2),
                                           ([1] * 4 + [33] + [1] * 8, 2), ([1, 1, 1, 40], 1), ([5, 5, 5], 1)])
@pytest.mark.parametrize("heads,e,n", [(2, 64, 128), (3, 10, 5), (2, 24, 300)])
def test_a_long_sequence_beside_single_tokens(k, heads, e, n, lens, launches, dtype):
    """A sequence's scan does not go token by token because the others bring one token each, and it gives what it gives alone."""
    g = torch.Generator(device=DEV).manual_seed(len(lens) + n)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    starts = [0]
    for m in lens:
        starts.append(starts[-1] + m)
    T, S = starts[-1], len(lens)
    xbc, dt = (rnd(T, heads * e + 2 * n) * 0.5).to(dtype), rnd(T, heads).to(dtype)
    dt_bias, a_log, skip, first = rnd(heads) - 1, rnd(heads), rnd(heads), rnd(S + 1, heads, e, n)
    slots = [(3 * i) % S if S % 3 else i for i in range(S)]

    def run(state, y, a, b):
        k.state_space_scan(xbc[starts[a]:starts[b]], dt[starts[a]:starts[b]], dt_bias, a_log, skip, state, y[starts[a]:starts[b]],
                           ints([s - starts[a] for s in starts[a:b + 1]]), ints(slots[a:b]), heads, 1, e, n)

    many, one = first.clone(), first.clone()
    y1, y2 = (torch.full((T, heads * e), float("nan"), device=DEV) for _ in range(2))
    before = k.launches
    run(many, y2, 0, S)
    assert k.launches - before == launches
    for i in range(S):
        run(one, y1, i, i + 1)
    # the same multiply-adds; a sum over the n rows in another order is n roundings of its magnitudes at most
    bound = lambda a: (n + 16) * 2.0 ** -24 * float(a.abs().max())
    assert float((y1 - y2).abs().max()) <= bound(y1) and float((one - many).abs().max()) <= bound(one)
    assert torch.equal(many[S], first[S])
