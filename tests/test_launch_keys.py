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
