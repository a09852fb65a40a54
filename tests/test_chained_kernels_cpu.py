"""Kernels that may start before the kernel ahead of them has ended (they call ``pdl_wait``) must not
read that kernel's output through the read-only path: ``__ldg`` and ``const __restrict__`` promise data
that is constant for the kernel's lifetime, and let the compiler move the load across the wait.

Nothing of it can be seen in the results of a run, so the sources are checked: what each of these
kernels and the functions it calls read that way has to be on the list below, with the reason why it
is complete before the kernel can start."""

import glob
import os
import re

import pytest

from moe_bench_b200 import build as mb_build

# The caller's tensors: written before a forward's first kernel, which is an ordinary launch.
CALLER = {"topk_ids", "expert_map", "args.w_scale", "args.row_scale", "src", "x"}
# The schedule, in the grouped GEMMs alone: their launch waits for the sort (ordinary launch), or is
# chained to a kernel (row gather, gate/up GEMM) that triggers only after its own wait has covered it.
SCHEDULE = {"counts", "args.sorted_ids"}
ALLOWED = {
    "align_count_kernel": CALLER,
    "align_scatter_kernel": CALLER,
    "combine_bf16_kernel": set(),
    "group_quant_fp8_kernel": CALLER,
    "gather_rows_peer_fp8_kernel": set(),
    "grouped_gemm_bf16_kernel": CALLER | SCHEDULE,
    "grouped_gemm_fp8_kernel": CALLER | SCHEDULE,
    "grouped_gemm_fp8_cols_kernel": CALLER | SCHEDULE,
}
# device functions these kernels call that load through the read-only path
CALLS = {"slot_of": CALLER, "decode_tile": SCHEDULE, "wait_limit_ns": {"status"}}


def _functions():
    """name -> (parameters, body) of every device function and kernel."""
    out = {}
    for path in sorted(glob.glob(os.path.join(mb_build.CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__(?:global|device)__[^;{}()]*(?:__launch_bounds__\([^)]*\)\s*)?\b(\w+)\(([^)]*)\)\s*(?:const\s*)?\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            out.setdefault(m.group(1), []).append((m.group(2), text[m.end() : i]))
    return out


FUNCTIONS = _functions()
CHAINED = sorted(n for n, v in FUNCTIONS.items() if any("pdl_wait()" in body for _, body in v))


def _read_only_loads(body):
    return {m.group(1) for m in re.finditer(r"__ldg\(\s*([\w.]+)", body)}


def test_the_kernels_are_known():
    assert set(CHAINED) | {"align_count_kernel"} == set(ALLOWED)
    loaders = {n for n, v in FUNCTIONS.items() if any("__ldg(" in b for _, b in v)}
    assert {"align_scatter_kernel", "combine_push_kernel", "decode_tile"} <= loaders | set(CHAINED)


@pytest.mark.parametrize("kernel", sorted(ALLOWED))
def test_only_finished_data_through_the_read_only_path(kernel):
    for params, body in FUNCTIONS[kernel]:
        assert _read_only_loads(body) <= ALLOWED[kernel]
        promised = set(re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params))
        assert promised <= {p.split(".")[-1] for p in ALLOWED[kernel]}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_their_device_functions(name):
    for _, body in FUNCTIONS[name]:
        assert _read_only_loads(body) <= CALLS[name]
    if name == "decode_tile":  # called by the grouped GEMMs only
        assert all("decode_tile(" not in b for k in ALLOWED if "gemm" not in k for _, b in FUNCTIONS[k])
