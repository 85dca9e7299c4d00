"""The recurrences over prompts, chunk by chunk: what a chunk may not do to the tokens before, and which calls it takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
RULES = ["delta", "decayed", "general"]


@pytest.fixture(scope="module")
def k():
    from chibillm_b200.kernels.ops import CudaKernels
    return CudaKernels(torch.device(DEV))


def ints(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


class Step:
    """A step's inputs, and its outputs and states under one of the three rules."""

    def __init__(self, k, rule, lens, heads, d, dtype=torch.float32, seed=0):
        self.k, self.rule, self.lens, self.heads, self.d = k, rule, lens, heads, d
        g = torch.Generator(device=DEV).manual_seed(d + seed)
        rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
        T, W = sum(lens), heads * d
        # r | k | v | gate | removal | low of the generalised rule, of which the others take the first three as q | k | v
        self.x, self.logits, self.beta = rnd(T, 5 * W + 8).to(dtype), rnd(T, W), rnd(T, heads).to(dtype)
        self.a_log, self.bias, self.removal = rnd(heads), rnd(W), rnd(W)
        self.decay = torch.rand(heads, generator=g, device=DEV)
        self.first = rnd(len(lens), heads, d, d)
        self.starts = [0]
        for n in lens:
            self.starts.append(self.starts[-1] + n)

    def run(self, longest=None):
        k, H, d, W = self.k, self.heads, self.d, self.heads * self.d
        state, o = self.first.clone(), torch.full((self.x.shape[0], W), float("nan"), device=DEV)
        q_start, slots, longest = ints(self.starts), ints(list(range(len(self.lens)))), longest or max(self.lens)
        if self.rule == "delta":
            k.channel_delta(self.x[:, :3 * W], self.logits, self.beta, self.a_log, self.bias, state, o, q_start, slots, H, H, d,
                            d, 1e-6, d ** -0.5, longest)
        elif self.rule == "decayed":
            k.decayed_attention(self.x[:, :3 * W], self.decay, state, o, q_start, slots, H, d, d, longest)
        else:
            k.delta_rule(self.x, self.logits, self.bias, self.removal, state, o, q_start, slots, H, d, 8, 0.6, 1e-6, longest)
        return o, state


# the chunk kernel's cuts: 8, 16 and 32 columns a block, 8 to 32 threads along the rows
@pytest.mark.parametrize("d,heads", [(20, 2), (20, 60), (64, 2), (64, 20), (64, 40), (128, 2), (128, 12), (128, 20), (200, 2), (200, 6),
                                     (200, 12)])
@pytest.mark.parametrize("rule", RULES)
def test_what_is_no_number_reaches_later_tokens_only(k, rule, d, heads):
    """One value, key, query, decay's logit or rate that is no number: the tokens before it, in its chunk of 16 and its tile of
    four too, and the other heads keep their bits."""
    step = Step(k, rule, [40], heads, d)
    clean, _ = step.run()
    assert torch.isfinite(clean).all()
    W, h = heads * d, heads - 1
    for at in (16, 21, 31):
        for part, what in enumerate(["query", "key", "value", None, "rate", "logit"]):
            if what is None or (rule != "general" and what == "rate") or (rule == "decayed" and what == "logit"):
                continue
            for bad in (float("nan"), float("inf")):
                where = step.logits[at] if what == "logit" else step.x[at]
                column = h * d + 3 + (0 if what == "logit" else part * W)
                kept = where[column].clone()
                where[column] = bad
                o, _ = step.run()
                where[column] = kept
                assert torch.equal(o[:at], clean[:at]), f"{bad} as token {at}'s {what} reached an earlier token"
                assert torch.equal(o[:, :h * d], clean[:, :h * d]), f"{bad} as token {at}'s {what} reached another head"
                if what != "logit" and bad != bad:
                    assert torch.isnan(o[at]).any()


@pytest.mark.parametrize("lens", [[40], [1, 33, 1, 1, 16, 17], [1] * 40 + [70] + [3] * 30])
@pytest.mark.parametrize("rule", RULES)
def test_the_longest_sequence_is_a_hint(k, rule, lens):
    """A number of tokens below that of the longest sequence picks no other chunks than the right one."""
    step = Step(k, rule, lens, 2, 64)
    right, wrong = step.run(), step.run(longest=5)
    assert torch.equal(right[0], wrong[0]) and torch.equal(right[1], wrong[1])


# sequences without a token, of single tokens, of whole chunks and a token more; 128 of them (what one look finds), one more or
# less, and many more
@pytest.mark.parametrize("lens", [[0, 16, 0, 0, 17, 1, 0], [1] * 31 + [50], [20] + [1] * 64 + [33], [1] * 126 + [50], [1] * 127 + [50],
                                  [1] * 128 + [50], [2] * 700 + [18] + [1] * 400])
@pytest.mark.parametrize("rule", RULES)
def test_every_sequence_of_a_mixed_step_gets_its_chunks(k, rule, lens):
    step = Step(k, rule, lens, 1, 32)
    o, state = step.run()
    for s in {0, 1, len(lens) // 2, len(lens) - 2, len(lens) - 1, max(range(len(lens)), key=lambda i: lens[i])}:
        a, b = step.starts[s], step.starts[s + 1]
        if a == b:
            assert torch.equal(state[s], step.first[s])
            continue
        alone = Step(k, rule, [b - a], 1, 32)
        alone.x, alone.logits, alone.beta, alone.first = step.x[a:b], step.logits[a:b], step.beta[a:b], step.first[s:s + 1]
        alone.a_log, alone.bias, alone.removal, alone.decay = step.a_log, step.bias, step.removal, step.decay
        # (the longest said to be five or more: chunks, as in the mixed step)
        one_o, one_state = alone.run(longest=max(5, b - a))
        assert torch.equal(o[a:b], one_o) and torch.equal(state[s:s + 1], one_state)


def test_a_decay_without_a_rank_is_refused(k):
    from chibillm_b200.kernels.ops import KernelError
    step = Step(k, "general", [1], 2, 32)
    W = 64
    with pytest.raises(KernelError):
        k.delta_rule(step.x[:, :5 * W], step.logits, step.bias, step.removal, step.first, torch.empty(1, W, device=DEV), ints([0, 1]),
                     ints([0]), 2, 32, 0, 0.6, 1e-6, 1)
