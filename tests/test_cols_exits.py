"""What a role of the register-block search kernel has in flight when it gives up
(csrc/cs_search_cols.cuh), read from the source: each bulk copy and each MMA is
waited for by the role that issued it, with a wait that another role's giving up
does not end, before the CTA's shared and tensor memory can go to the next one."""
import os
import re

from conftest import ROOT

SRC = open(os.path.join(ROOT, "coherentsearch_c_b200", "csrc", "cs_search_cols.cuh")).read()
KERNEL = SRC[SRC.index("search_cols(const __grid_constant__"):]


def role(start, end):
    return KERNEL[KERNEL.index(start):KERNEL.index(end)]


def test_box_warps_wait_for_their_copies():
    text = role("window boxes:", "the chunk and active harmonics")
    loop, leave = text[:text.index("never leave with copies")], text[text.index("never leave with copies"):]
    issued = set(re.findall(r"bulk_in\([^;]*?(\w+)\);", loop)) | \
        set(re.findall(r"tma_rows\([^;]*?(\w+)\);", loop))
    names = {"b": "wfull"}                          # b is a stage's wfull
    assert issued == {"tbar", "b"}
    for bar in issued:
        assert re.search(r"mbar_wait\(%s\b" % names.get(bar, bar), leave), bar
    assert "full_wait(" not in leave                # that one ends when any role gives up


def test_mma_warp_waits_for_its_mmas():
    """After the tile loop, on every way out of it: a commit behind all that was
    issued, and a wait for it; the operand images are waited for too."""
    text = role("--- MMAs ---", "tmem_dealloc")
    leave = text[text.index("never leave with"):]
    assert re.search(r"mma_commit\(drain\);\s*landed = mbar_wait\(drain, 0\)", leave)
    assert "mbar_wait(bbar, 0)" in leave
    before = text[:text.index("never leave with")]
    assert before.rstrip().endswith("/*") and "if (!ok) {" not in before    # not only where it failed
