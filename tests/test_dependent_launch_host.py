"""A launch behind a dependent launch waits for that grid alone, and a grid is over once its blocks have left. So that a wait
covers everything in front, the first block of every dependent grid waits (griddepcontrol.wait) on every path before it leaves:
the early returns in the source. And no load is allowed to move up across the wait. No run could show a violation, the grids'
overlap is a matter of timing."""
import os
import re

import pytest

from conftest import ROOT
from test_cluster_start_host import CSRC, _kernels

WAIT = re.compile(r"griddepcontrol\.wait|\bpdl_wait\(|\bms_begin\(|\bhad_tiled_begin\(")
# Early returns that the first block never takes
NOT_FIRST = {
    "gemv_prerotate_kernel": {"if (task >= m * per_row) return;"},
    "exl3_gemv_tc_kernel": {"if (cta >= ncta) return;"},     # (its work is known on the host, and not empty)
    "exl3_gemv_kernel": {"if (u0 >= u1) return;", "if (cblk * G >= U) return;"},       # behind cta >= ncta: the first of ncta ranges is not empty
    # (a CTA whose expert has another bit width: such launches are not dependent)
    "exl3_gemm_tc_kernel": {"if (bits && bits[P.g_tile_e[blockIdx.y]] != K) return;"},
}


def _early_returns(body):
    """Every return of a kernel (not of a lambda in it) in front of its last wait: the if statement or block that it ends"""
    last = max((m.start() for m in WAIT.finditer(body)), default=0)
    blocks = []                                              # (start of the statement that opens a block, inside a lambda)
    for m in re.finditer(r"[{}]|\breturn;", body[:last]):
        at = m.start()
        if m.group() == "}":
            blocks.pop()
            continue
        start = max(body.rfind(c, 0, at) for c in ";{}") + 1
        if m.group() == "{":
            blocks.append((start, bool(blocks and blocks[-1][1]) or bool(re.search(r"\[&\][^;{}]*$", body[start:at]))))
        elif not (blocks and blocks[-1][1]):
            if not re.match(r"\s*if\b", body[start:at]):
                start = blocks[-1][0]                        # last statement of a block: from its condition on
            yield " ".join(body[start:m.end()].split())


DEPENDENT = [(name, kernel, body) for name in sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
             for kernel, body in _kernels(name) if WAIT.search(body)]


@pytest.mark.parametrize("name,kernel", [d[:2] for d in DEPENDENT])
def test_first_block_waits_before_it_leaves(name, kernel):
    body = next(b for n, k, b in DEPENDENT if (n, k) == (name, kernel))
    for statement in _early_returns(body):
        assert WAIT.search(statement) or statement in NOT_FIRST.get(kernel, ()), statement


def test_nothing_in_front_of_the_wait_is_declared_unaliased():
    """A load through a const __restrict__ pointer may be moved across the wait (the compiler takes what it points to as constant
    for the whole kernel): only static operands are declared so in a dependent kernel."""
    kernels = {k for _, k, _ in DEPENDENT}
    seen = set()
    for name in sorted({n for n, _, _ in DEPENDENT}):
        text = re.sub(r"/\*.*?\*/|//[^\n]*", "", open(os.path.join(CSRC, name)).read(), flags=re.S)
        for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\(([^)]*)\)\s*\{", text):
            if m.group(1) in kernels:
                seen.add(m.group(1))
                assert set(re.findall(r"__restrict__\s+(\w+)", m.group(2))) <= {"suh", "t_suh", "w"}, m.group(1)
    assert seen == kernels


def test_the_search_finds_the_kernels():
    found = {k for _, k, _ in DEPENDENT}
    assert found >= {"exl3_gemv_kernel", "exl3_gemv_tc_kernel", "exl3_gemm_tc_kernel", "moe_prep_kernel", "moe_sorted_combine_kernel",
                     "had_tiled_kernel", "had_tiled_rows_kernel", "gemv_prerotate_kernel"}
