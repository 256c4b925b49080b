"""Hand-overs of the tensor-core kernels, checked on the CPU from their source (a missing wait or fence rarely shows in an output)."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "lfm2-ampere_b200" / "csrc"

# a wait, the fence that orders tcgen05 operations behind it, and the operations themselves
TOKEN = re.compile(r"(?P<open>\{)|(?P<close>\})|(?P<wait>\btc_wait(?:<\w+>)?\()|(?P<fence>\btc_fence_after\()"
                   r"|(?P<op>\btc_(?:ld\d*(?:<[^>]*>)?|st8|mma_\w+)\()")


def unfenced(text):
    """Lines of tcgen05 operations that some path reaches from a barrier wait without tcgen05.fence::after_thread_sync between
    the two.  A fence inside a block counts for that block alone: the block may be skipped."""
    text = re.sub(r"//[^\n]*", "", text)
    bad, due, blocks, before = [], False, [], False
    for t in TOKEN.finditer(text):
        if t["open"]:                                    # (state on entry, state at the end of the branches before this one)
            blocks.append((due, before))
            before = False
        elif t["close"]:
            entry, earlier = blocks.pop()
            if text[t.end():t.end() + 8].lstrip().startswith("else"):
                before, due = earlier or due, entry
            else:
                due = due or entry or earlier
        elif t["wait"]:
            due = True
        elif t["fence"]:
            due = False
        elif due:
            bad.append(text.count("\n", 0, t.start()) + 1)
    return bad


def test_checker_sees_a_fence_that_may_be_skipped():
    assert unfenced("f() { tc_wait(b); if (grown) { tc_fence_after(); tc_ld8(o); } tc_st8(p); }") == [1]
    assert unfenced("f() { tc_wait(b); tc_fence_after(); if (grown) { tc_ld8(o); } tc_st8(p); }") == []
    assert unfenced("f() { if (producer) { tc_wait(b); } else { tc_ld8(o); } tc_st8(p); }") == [1]


@pytest.mark.parametrize("name", ["lkb_pfattn.cu", "lkb_gemm_tc.cu"])
def test_every_tmem_access_is_fenced_behind_its_wait(name):
    assert unfenced((CSRC / name).read_text()) == []
