"""Waits of the kernels on counters that other blocks raise.

A kernel reads rows that other blocks wrote once it has acquired their counters, a counter per lane.
What a lane has acquired is ordered for that lane alone; the vote that tells the others orders no
memory (``__syncwarp`` does), and ``elect.sync`` leaves open which lane issues the loads.

A stale row needs an unlucky moment that no run can be made to show, so the sources are checked."""

import glob
import os
import re

import pytest

from moe_bench_b200 import build as mb_build

GEMMS = ("grouped_gemm.cu", "grouped_gemm_fp8.cu", "grouped_gemm_fp8_cols.cu")


def _source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(mb_build.CSRC, name)).read())


def _block(text, start):
    """The text from the first brace at or after `start` to the brace that closes it."""
    i = text.index("{", start)
    depth, j = 1, i + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
    return text[i:j]


def test_the_lanes_acquires_are_joined_before_the_wait_returns():
    common = _source("common.cuh")
    body = _block(common, common.index("bool wait_counters("))
    poll = _block(body, body.index("while (true)"))
    assert "ld.acquire.gpu" in poll
    after = body[body.index(poll) + len(poll) :]
    assert re.fullmatch(r"\s*__syncwarp\(\);\s*return true;\s*}", after)


@pytest.mark.parametrize("name", GEMMS)
def test_a_vote_is_not_what_orders_the_rows(name):
    """No wait of its own that acquires a counter per lane, and none but that wait ahead of a proxy fence."""
    text = _source(name)
    assert not re.search(r"if \(lane < [^;{}]*\)\s*asm volatile\(\"ld\.acquire", text)
    for m in re.finditer(r"fence\.proxy\.async;", text):
        assert re.search(r"ok = wait_counters<[^;]*;\s*if \(!ok\) break;\s*asm volatile\(\"$", text[: m.start()])


def test_the_kernels_that_wait_for_rows_are_known():
    waits = {os.path.basename(p) for p in glob.glob(os.path.join(mb_build.CSRC, "*.cu")) if "fence.proxy.async" in _source(os.path.basename(p))}
    assert waits == {"grouped_gemm.cu", "grouped_gemm_fp8.cu"}


@pytest.mark.parametrize("name", GEMMS)
def test_one_thread_issues_all_loads_of_a_barrier(name):
    """Every call that arms a stage's barrier or loads into it is behind the same choice of a lane."""
    text = _source(name)
    calls = [m.start() for m in re.finditer(r"\bload_weights\(kb", text)]
    assert len(calls) == 2
    guards = {re.findall(r"if \((lane == 0|elect_one\(\))\)", text[:at])[-1] for at in calls}
    assert len(guards) == 1


@pytest.mark.parametrize("name", GEMMS)
def test_no_lane_leaves_a_polling_loop_alone(name):
    """A lane that breaks out on what it read itself would be missing from the full-mask votes of the
    lanes that read the counter a moment earlier: all polling is done by the wait whose exit is a vote."""
    assert "ld.acquire" not in _source(name)
    common = _source("common.cuh")
    body = _block(common, common.index("bool wait_counters("))
    assert re.findall(r"if \(([^;{}]*)\) break;", body) == ["__all_sync(0xffffffffu, v >= target)"]
