"""Rules that the kernels' sources keep and that no single run can show."""
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc", "src", "kernels")


def _overlapped():
    """The sources of kernels that are launched while the kernel in front of them runs, each with the headers it takes from here."""
    found = {}
    for name in sorted(os.listdir(KERNELS)):
        text = open(os.path.join(KERNELS, name)).read()
        if name.endswith(".cu") and "kernels/programmatic_launch.cuh" in text:
            found[name] = [name] + [h for h in re.findall(r'#include "kernels/([^"]+)"', text) if os.path.exists(os.path.join(KERNELS, h))]
    return found


@pytest.mark.parametrize("kernel", sorted(_overlapped()))
def test_overlapped_kernels_load_coherently(kernel):
    """The read-only path is for data that stays as it is for as long as the kernel runs.  The kernel in front of an overlapped
    launch may still write what it loads, and a read-only load is not tied to the wait for that kernel either."""
    assert len(_overlapped()) >= 5
    for name in _overlapped()[kernel]:
        code = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(KERNELS, name)).read(), flags=re.S)
        assert not re.findall(r"__ldg\b|__restrict__|ld\.global(?:\.\w+)*\.nc\b", code), name
        assert "waitForPreviousKernel" in code or not name.endswith(".cu")


def test_scale_rows_change_hands_between_tiles():
    """A promotion warp with swapped operands shares its scales through two rows of shared memory, step by step in turn.  With an odd
    number of steps a tile begins with the row that the tile before ended with: the warp has to meet before that is written."""
    code = re.sub(r"//[^\n]*", "", open(os.path.join(KERNELS, "grouped_gemm_fp8.cu")).read())
    body = code[code.index("bool promoteSwapped(") :]
    body = body[: body.index("\n}\n")]
    row = re.search(r"scales\[(.*?)\]\[lane\] =", body).group(1)
    used = [eval(row, {"j": step % 4}) for tile in range(2) for step in range(3)]
    again = [i for i in range(1, len(used)) if used[i] == used[i - 1]]
    assert again == [3]  # the second tile's first step, and no other
    assert "__syncwarp()" in body[: body.index("for (int ks0")]


@pytest.mark.parametrize("kernel", sorted(_overlapped()))
def test_overlapped_kernels_fetch_nothing_by_guess(kernel):
    """In front of the wait for the previous kernel nobody knows what will be read (the routing is what that kernel writes): expert
    weights that were called into L2 there by their place were read in vain wherever the first experts had no rows."""
    code = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(KERNELS, kernel)).read(), flags=re.S)
    for begin in re.finditer(r"__global__", code):
        body = code[begin.start() :].split("__global__", 2)[1]
        ahead, wait, _ = body.partition("waitForPreviousKernel()")
        assert not wait or "prefetch" not in ahead


@pytest.mark.parametrize("kernel", sorted(_overlapped()))
def test_overlapped_kernels_without_shared_memory_ask_for_l1(kernel):
    """An SM that a GEMM has just left has hardly any L1 unless the kernel that moves in asks for it."""
    code = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(KERNELS, kernel)).read(), flags=re.S)
    for begin in re.finditer(r"nixl_pdl::launch\(kernel, [^;]*?, 0, ", code):
        assert "nixl_pdl::preferL1(" in code[code.rindex("const auto kernel", 0, begin.start()) : begin.start()]
