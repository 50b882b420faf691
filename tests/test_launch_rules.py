"""Rules of the sources that no run can show to be kept: every kernel here may be resident while the one
before it in the stream still writes (programmatic dependent launch), so what other kernels write is
not read through the read-only path, which is for data that nobody writes meanwhile."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "chatokf_b200" / "csrc"


def code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def kernels(name):
    """(head, body) of every kernel of a source file."""
    text = code(name)
    for m in re.finditer(r"__global__[^{;]*\{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(0), text[m.end():at]


@pytest.mark.parametrize("name", ["okf_gemv.cu", "okf_gemm_tc.cu", "okf_gemm_ts.cu", "okf_neighbours.cu"])
def test_results_of_other_kernels_are_not_read_through_the_read_only_path(name):
    found = [(h, b) for h, b in kernels(name) if "pdl_wait" in b]
    assert found
    for head, body in found:
        read_only = re.findall(r"const\s+(\w+)\s*\*\s*__restrict__\s*(\w+)", head)
        assert set(read_only) <= {("uint8_t", "w")}, head  # weights
        assert "__ldg(" not in body, head
    if name == "okf_gemv.cu":  # x is staged by functions of their own
        assert "__ldg(" not in code(name)


def test_a_ring_stage_is_handed_back_only_when_its_words_have_been_used():
    """The copy that refills a stage of the prefill matmul's ring waits for the unpacking warps' arrivals and for nothing
    else: they come behind the last instruction that needs a word loaded from the stage."""
    (head, body), = [(h, b) for h, b in kernels("okf_gemm_ts.cu") if "empty_w" in b]
    arrivals = [m.start() for m in re.finditer(r"mbar_arrive\(&empty_w", body)]
    assert len(arrivals) == 1
    for use in ("raw.load(", "unpack<F16>(", "tmem_st32("):
        at = [m.start() for m in re.finditer(re.escape(use), body)]
        assert at and max(at) < arrivals[0], use
    between = body[max(at):arrivals[0]]
    assert between.count("}") >= between.count("{") + 2, "behind the loop over k-blocks"


def test_a_warp_whose_first_lane_waits_is_ordered_behind_that_wait():
    """Bytes that a barrier hands over are seen by the thread that waited on it and by those it synchronises with
    afterwards; a shuffle is no such synchronisation."""
    waits = {"okf_tc.cuh": 1, "okf_gemv.cu": 1, "okf_gemm_tc.cu": 0, "okf_gemm_ts.cu": 0}
    for name, count in waits.items():
        found = list(re.finditer(r"lane == 0[^;]*\bmbar_wait\w*\(", code(name)))
        assert len(found) == count, name
        for m in found:  # before anything is copied or read, and before the function that waits is left
            rest = code(name)[m.end():]
            touched = re.search(r"bulk_g2s\(dst \+|return ok;|\n    \};", rest)
            assert touched and "__syncwarp();" in rest[:touched.start()], name
