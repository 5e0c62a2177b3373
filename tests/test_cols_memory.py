"""What the register-block search keeps for itself may not cost a call its memory
(csrc/cs_gpu.cu, read from the source, since a full device is no test's to make): it
is allocated after every buffer that a session needs, and a record buffer that cannot
grow takes its place."""
import os
import re

from conftest import ROOT

SRC = open(os.path.join(ROOT, "coherentsearch_c_b200", "csrc", "cs_gpu.cu")).read()


def body(head):
    text = SRC[SRC.index(head):]
    return text[:text.index("\n}\n")]


def test_it_is_the_last_buffer_of_a_session():
    load = body("static int session_load(")
    allocs = [m.start() for m in re.finditer(r"dev_reserve\(|cudaMalloc\(|grow_records\w*\(|"
                                             r"t(?:ci|ma)_load\(", load)]
    assert len(allocs) > 12
    assert load.index("cols_load(") > max(allocs)


def test_records_take_its_place():
    grow = body("static int grow_records(")
    first = grow.index("cudaMalloc(")
    assert first < grow.index("cols_drop(") < grow.index("cudaMalloc(", first + 1)
    drop = body("static bool cols_drop(")
    for left in ("d_cols = NULL", "c_cols = 0", "use_cols = 0"):
        assert left in drop


def test_wide_fp64_search_does_without_its_weights():
    load = body("static int session_load(")
    at = load.index("dev_reserve((void **)&S->d_wt64")
    assert "CK(" not in load[at - 40:at] and "S->f64_wide = 0" in load[at:at + 400]
