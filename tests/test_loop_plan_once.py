"""A loop call reads the autotuner's choice once: any thread may tune or pin a side while
another enqueues its passes, and passes of one call on different plans would take packed tiles
of another width and leave out different columns.  Checked in the sources (no GPU)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ctdm_gb300", "csrc")


def body(name, signature):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    start = text.index("{", re.search(signature, text).end() - 1)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i]


def test_launches_take_the_callers_plan():
    for fn in ("plane", "xpass", "ypass", "zpass"):
        b = body("tune.cu", r"cudaError_t launch_%s\([^)]*\)\s*\{" % fn)
        assert not re.search(r"choice_of|loop_scheme|loop_plan|g_choice", b), fn


def test_one_read_per_call():
    b = body("ctdm_api.cu", r"static ctdm_status do_positivity\([^{;]*\)\s*\{")
    assert len(re.findall(r"\bloop_plan\(", b)) == 1
    assert not re.search(r"loop_scheme\(|loop_ztile\(|choice_of", b)
