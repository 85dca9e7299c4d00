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
    spec = SimpleNamespace(num_heads=32, num_kv_heads=8, head_dim=head_dim)
    runtime = Runtime(torch.device("cpu"), dtype, kernels)
    paged = SimpleNamespace(position=SimpleNamespace(fused_rotation=lambda: True), runtime=runtime, spec=spec, prepared=False,
                            maps=1, value_dim=head_dim)
    latent = SimpleNamespace(runtime=runtime, spec=spec, key_dim=head_dim)
    steps = [SimpleNamespace(num_seqs=8, max_ctx_len=n) for n in (1, 64, 65, 128, 129, 256, 257, 500, 1000, 2047, 2048, 4096, 9000)]
    assert len({PagedAttention.launch_key(paged, c) for c in steps}) == captures
    if dtype == torch.float32:
        assert len({LatentAttention.launch_key(latent, c) for c in steps}) == captures
