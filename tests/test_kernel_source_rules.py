"""Rules that the kernels keep by the order or the kind of their instructions, and that no run can be made to show."""
import os
import re

import fused_attention_b200 as fa

CSRC = os.path.join(os.path.dirname(fa.__file__), "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def body_behind_the_wait(name, kernel):
    text = source(name)
    text = text[text.index(f"\n{kernel}("):]
    return text[text.index("grid_dep_wait();"):]


def test_a_launch_without_work_asks_for_no_copies():
    """A kernel that stands behind a planned one reads whether that one took the call before its first copy: with nothing
    to do no role waits for a copy, and the CTA would leave with it still landing in shared memory."""
    for name, kernel in (("fa_kernels.cuh", "fa_fwd_pipelined"), ("fa_pair.cuh", "fa_fwd_pair")):
        text = body_behind_the_wait(name, kernel)
        assert text.index("p.plan_head") < re.search(r"\b(load_tile|tma_load_3d)\w*[<(]", text).start(), kernel


def test_no_load_of_read_only_data():
    """Every kernel may be resident while the kernel before it still writes: what it loads is not read-only for its life,
    which ld.global.nc asks for, and such a load need not stay behind the wait for that kernel."""
    names = [n for n in os.listdir(CSRC) if n.endswith((".cu", ".cuh"))]
    assert names and not [n for n in names if re.search(r"__ldg\b|ld\.global\.nc", source(n))]


def test_the_plan_counts_its_ctas_in_a_word_of_its_own():
    """The part counters of divided calls can be left half counted by a launch that gave up, and are zeroed with its
    report at any time; a plan that counted there would never find its last CTA and leave old lists in place."""
    text = source("fa_b200.cu")
    assert re.search(r"a\.ticket = scratch\.ticket;", text)
    report = text[text.index("int fold_ctx_status"):text.index("uint32_t next_launch_id")]
    assert "ticket" not in report and ".cnt" in report
