"""The give-up path of the kernels' bounded waits, read from the sources: a wait that runs out must not leave a part of a
warp, or some of the warps, behind at a vote or a barrier that the rest never comes to.  (A wait cannot be made to run out
inside a kernel of many warps without a broken pipeline, which no test runs on a GPU.)"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "ziglm_b200", "csrc")
FILES = ["attention_fmha.cu", "attention_tc.cu", "gemm_generic.cu", "gemm_tc.cu", "tc_common.cuh"]
ONE_LANE = re.compile(r"\blane == 0\b|\bthreadIdx\.x == 0\b")


def uses(text, pattern):
    """(line, statement up to the use, headers of the blocks around it) of every use of ``pattern`` outside comments."""
    text = re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), text)
    hits = [m.start() for m in re.finditer(pattern, text)]
    stack, begin, found, k, depth = [], 0, [], 0, 0
    for i, c in enumerate(text):
        if k < len(hits) and i == hits[k]:
            found.append((text.count("\n", 0, i) + 1, text[begin:i], list(stack)))
            k += 1
        depth += (c == "(") - (c == ")")
        if c == "{":
            stack.append(text[begin:i])
        elif c == "}":
            stack.pop()
        if c in "{}" or (c == ";" and depth == 0):
            begin = i + 1
    return found


def one_lane(statement, headers):
    return any(ONE_LANE.search(h) for h in headers + [statement])


@pytest.mark.parametrize("name", FILES)
def test_a_warp_that_branches_on_a_wait_branches_as_one(name):
    """A plain mbar_wait answers each lane by itself: it stands where one lane runs alone, or in the functions that make
    one answer of it, or where nothing depends on the answer."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    for line, statement, headers in uses(text, r"(?<!\w)mbar_wait\("):
        if one_lane(statement, headers):
            continue
        if "__all_sync(" in statement:
            continue
        if not headers or re.search(r"\bbool $", statement.split("\n")[-1]):       # its own definition
            continue
        if any("produce_pages(" in h for h in headers):                            # called by one lane, see below
            continue
        unused = re.fullmatch(r"\s*(if \(n_kb > 0\)\s*)?", statement)
        assert unused, f"{name}:{line}: the lanes of a warp may take different ways: {statement.strip()}"
    for line, statement, headers in uses(text, r"produce_pages<"):
        assert one_lane(statement, headers), f"{name}:{line}"


@pytest.mark.parametrize("name", FILES)
def test_warps_that_meet_at_barriers_read_the_abort_flag_as_one(name):
    """The flag may be set between two warps' reads of it: what several warps do next is decided by a barrier that ORs what
    they read.  A read stands where one lane runs alone, in such a barrier, or where the warp only returns."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    for line, statement, headers in uses(text, r"\*abort_flag\b(?!\s*=[^=])"):
        if one_lane(statement, headers) or any("mbar_wait(" in h or "produce_pages(" in h for h in headers):
            continue
        if re.search(r"\bbar_(consumers_)?or(<[^>]*>)?\($", statement):
            continue
        after = text.splitlines()[line - 1].split("*abort_flag", 1)[1]
        assert re.match(r"\) return;", after), f"{name}:{line}: warps may decide differently: {statement.strip()}"


def test_prompt_attention_asks_for_no_more_registers_than_a_build_has():
    """The prompt attention's warps share out again what a block was launched with; asking for more than that waits for good.
    A build of fewer registers a thread than the split needs is refused before the launch (the caller has another kernel)."""
    from ziglm_b200 import csrc
    fit = csrc.load("attention_fmha").zlm_attention_fmha_shares_fit
    assert fit(168) == 1
    assert fit(160) == 0 and fit(128) == 0
    with open(os.path.join(CSRC, "attention_fmha.cu")) as f:
        launch = f.read().split("static int fm_launch(", 1)[1]
    assert launch.index("fm_shares_fit(built.numRegs)") < launch.index("launch_pdl(")
