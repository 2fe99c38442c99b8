"""Waits of the warps that issue tcgen05 instructions, read from the kernels' source: nothing here can be tried on a GPU without hanging it.

Such a warp elects a lane with elect.sync, which needs every lane of the warp.  A wait that each lane ends by its own clock lets the
lanes disagree when a barrier completes around the limit: those that gave up leave, the others stand in elect.sync.  So a wait
has one answer for the warp (tc_wait_warp), in every role that elects."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "skainet_b200", "csrc")


def roles(text):
    """Bodies of the outermost `if (warp ...) {` blocks that hold a tc_elect()."""
    text = re.sub(r"//[^\n]*", "", text)
    found, open_at = {}, []
    for at, ch in enumerate(text):
        if ch == "{":
            head = text[max(text.rfind(c, 0, at) for c in ";{}") + 1:at]
            open_at.append((at, bool(re.search(r"if \(warp\b", head))))
        elif ch == "}":
            open_at.pop()
        elif text.startswith("tc_elect()", at):
            role = next((p for p, is_role in open_at if is_role), None)
            if role is not None:
                found[role] = None
    for p in found:
        depth = 0
        for at in range(p, len(text)):
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            if depth == 0:
                found[p] = text[p:at]
                break
    return list(found.values())


@pytest.mark.parametrize("name", ["skn_dense.cu", "skn_matmul_tc.cu", "skn_matvec_batch.cu"])
def test_a_warp_that_elects_waits_as_one(name):
    with open(os.path.join(CSRC, name)) as f:
        blocks = roles(f.read())
    assert blocks, "no issuing role found"
    for body in blocks:
        assert "tc_wait_warp(" in body
        assert "skn_mbar_wait(" not in body


@pytest.mark.parametrize("name", ["skn_dense.cu", "skn_matmul_tc.cu", "skn_matvec_batch.cu"])
def test_tensor_memory_is_touched_behind_a_fence(name):
    """Stores to tensor memory, loads from it and MMAs follow the barrier that they wait for only through tcgen05.fence::after_thread_sync: it
    stands between every access and the wait before it."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    waited, accesses = None, 0
    for m in re.finditer(r"(tc_wait_warp|skn_mbar_wait)\(|(tc_fence_after)\(|(?<!void )\b(tc_(?:ld|st)(?:8|16|32)\w*|tc2?_mma_\w+)\(", text):
        if m[1]:
            waited = m.start()
        elif m[2]:
            waited = None
        else:
            accesses += 1
            assert waited is None, f"{m[3]} at line {text.count(chr(10), 0, m.start()) + 1}, no fence since the wait at line {text.count(chr(10), 0, waited) + 1}"
    assert accesses >= 2
