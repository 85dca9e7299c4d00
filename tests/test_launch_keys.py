"""What a captured step's key holds: what the host decides for its kernels, and nothing else."""
from types import SimpleNamespace

import pytest
import torch

from chibillm_b200.kernels.ops import CudaKernels
from chibillm_b200.parts.base import Runtime


@pytest.mark.parametrize("head_dim,dtype,differs", [(64, torch.float32, True), (128, torch.float32, True), (80, torch.float32, False),
                                                    (192, torch.float32, False), (128, torch.bfloat16, False)])
def test_32_bit_attention_is_captured_anew_only_where_its_kernels_depend_on_the_context(head_dim, dtype, differs):
    """Head sizes of the kernel whose CTAs share a token's keys: one capture for each number of CTAs.  Others run the plain
    kernel (or bfloat16's own): one capture whatever the contexts."""
    runtime = Runtime(torch.device("cpu"), dtype, CudaKernels)
    keys = [runtime.float32_launch_key(SimpleNamespace(max_ctx_len=n), head_dim) for n in (1, 64, 65, 128, 129, 256, 257, 5000)]
    assert len(set(keys)) == (4 if differs else 1)
    assert all(len(k) == (1 if differs else 0) for k in keys)


def test_a_question_about_scratch_is_no_launch():
    """The table of launches (--profile) has no line for an entry point that only answers."""
    from chibillm_b200.kernels import profile
    assert "chibi_recurrence_scratch" in profile._NOT_LAUNCHES


@pytest.mark.parametrize("head_dim,dtype,captures", [(64, torch.float32, 4), (128, torch.float32, 4), (80, torch.float32, 1),
                                                     (128, torch.bfloat16, 5)])
def test_attention_is_captured_anew_only_for_what_its_own_kernels_depend_on(head_dim, dtype, captures):
    """The bfloat16 kernel's key ranges and how they are cut (eight sequences: one to four ranges, by length from 2,048 keys
    on) are nothing to the 32-bit kernels."""
    from chibillm_b200.parts.attention import PagedAttention
    from chibillm_b200.parts.latent_attention import LatentAttention
    kernels = CudaKernels.__new__(CudaKernels)
    kernels.sm_count = 148
    spec = SimpleNamespace(num_heads=32, num_kv_heads=8, head_dim=head_dim, window=None, chunk=None)
    runtime = Runtime(torch.device("cpu"), dtype, kernels)
    paged = SimpleNamespace(position=SimpleNamespace(fused_rotation=lambda: True), runtime=runtime, spec=spec, prepared=False,
                            maps=1, value_dim=head_dim)
    latent = SimpleNamespace(runtime=runtime, spec=spec, key_dim=head_dim)
    steps = [SimpleNamespace(num_seqs=8, max_ctx_len=n, even_contexts=lambda *a: False) for n in (1, 64, 65, 128, 129, 256, 257, 500, 1000, 2047, 2048, 4096, 9000)]
    assert len({PagedAttention.launch_key(paged, c) for c in steps}) == captures
    if dtype == torch.float32:
        assert len({LatentAttention.launch_key(latent, c) for c in steps}) == captures


def _context(ctx_lens, q_lens=None):
    from chibillm_b200.engine.batch import StepContext
    from dataclasses import fields
    c = StepContext(**{f.name: None for f in fields(StepContext)})
    c.shared, c.ctx_lens, c.q_lens = {}, ctx_lens, q_lens or [1] * len(ctx_lens)
    c.num_seqs, c.max_ctx_len = len(ctx_lens), max(ctx_lens)
    return c


@pytest.mark.parametrize("lens,q_lens,window,chunk,even", [
    ([2048] * 8, None, None, None, True), ([2048] * 7 + [1], None, None, None, True), ([2048] * 6 + [1, 1], None, None, None, False),
    ([4096, 1024], None, None, None, False), ([4096, 1024], None, 1000, None, True), ([4096, 1024, 10], None, 1000, None, False),
    ([1024 * 4, 1024 * 2], None, None, 1024, True), ([1024 * 4, 1024 * 2 + 1], None, None, 1024, False),
    ([2000, 2000, 9], [1, 1, 9], None, None, True), ([9000, 9], [9000, 9], None, None, True)])
def test_even_contexts(lens, q_lens, window, chunk, even):
    """What the single tokens of a step see: an eighth less than the most on average is still even."""
    assert _context(lens, q_lens).even_contexts(window, chunk) is even


def test_even_steps_are_shared_out_without_their_lengths():
    kernels = CudaKernels.__new__(CudaKernels)
    kernels.sm_count = 148
    assert kernels.decode_attention_key(8, 32, 8, 4096, True) == (4, 0, 0)
    assert kernels.decode_attention_key(8, 32, 8, 4096) == (4, 37, 0)
    assert kernels.decode_attention_key(64, 32, 8, 4096, True)[1:] == (0, 0) and kernels.decode_attention_key(64, 32, 8, 4096) == (1, 0, 1)
