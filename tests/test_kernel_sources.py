"""What the CUDA sources must keep to and no run on a GPU may show (a wait that runs out, for one)."""
import os
import re

import pytest

import chibillm_b200.csrc

CSRC = os.path.dirname(chibillm_b200.csrc.__file__)


def lone_waits(text):
    """Lines where lanes decide one by one by the outcome of a wait, outside a block that one thread alone runs."""
    text = re.sub(r"//[^\n]*", "", text)
    found, headers, at = [], [], 0               # headers: what stands before each open brace
    for m in re.finditer(r"[{}]|\bmbar_wait(?:_warp)?\(", text):
        if m.group() == "{":
            headers.append(re.split(r"[;{}]", text[:m.start()])[-1])
        elif m.group() == "}":
            headers.pop()
        elif m.group() == "mbar_wait(":
            before = re.split(r"[;{}]", text[:m.start()])[-1].strip()
            alone = any("elect_one()" in h or "lane == 0" in h or "threadIdx.x == 0" in h for h in headers)
            plain = before == "" or re.fullmatch(r"(if|else if|for) \(.*\)|else", before, re.S)      # nobody looks at the outcome
            if not plain and not alone:
                found.append(text[:m.start()].count("\n") + 1)
    return found


def test_the_check_sees_a_lane_that_leaves_by_itself():
    assert lone_waits("void f() {\n  if (warp > 1) {\n    if (!mbar_wait(b, 0, e, 1))\n      break;\n  }\n}") == [3]
    assert lone_waits("void f() {\n  const bool ok = mbar_wait(b, 0, e, 1);\n}") == [2]
    assert lone_waits("void f() {\n  if (elect_one()) {\n    if (!mbar_wait(b, 0, e, 1))\n      break;\n  }\n}") == []
    assert lone_waits("void f() {\n  if (j >= 2)\n    mbar_wait(b, 0, e, 1);\n  if (!mbar_wait_warp(b, 0, e, 1))\n    return;\n}") == []


@pytest.mark.parametrize("name", sorted(n for n in os.listdir(CSRC) if n.endswith(".cu")))
def test_a_wait_that_runs_out_is_a_whole_warps(name):
    with open(os.path.join(CSRC, name)) as f:
        assert lone_waits(f.read()) == []


def test_the_recurrences_ask_for_their_shared_memory_whatever_its_size():
    """A block has 48 KB without asking, its kernel's own arrays among them (general_prepare_kernel's 6 KB beside 42 KB for heads of
    128, and a word more in a timeline build): the dynamic part alone does not tell."""
    with open(os.path.join(CSRC, "linear_recurrence.cu")) as f:
        text = f.read()
    assert not re.findall(r"if \(smem > [^)]*\)", text)
    assert text.count("if (const int e = allow_shared(") == 2          # the preparing kernels and the chunk kernels


@pytest.mark.parametrize("name", sorted(n for n in os.listdir(CSRC) if n.endswith((".cu", ".cuh"))))
def test_rules_ask_the_device_for_its_sms(name):
    with open(os.path.join(CSRC, name)) as f:
        assert not re.findall(r"constexpr[^;]*\b148\b", re.sub(r"//[^\n]*", "", f.read()))
