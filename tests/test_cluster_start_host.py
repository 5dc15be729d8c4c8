"""Every kernel that accesses another CTA's shared memory first makes sure that the CTA runs (the CUDA programming model
guarantees a peer's shared memory only from then on): the order of arrival, wait and first access in the source. No run
could show a violation, a peer that starts late is a matter of timing."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "ampstein_b200", "csrc")
ACCESS = re.compile(r"\bcluster_st_f32\(|\bmp_ld_cluster\(|\btg_st_cluster_u32\(")


def _kernels(name):
    """(kernel name, body) of every __global__ function of a source file, comments removed"""
    text = re.sub(r"/\*.*?\*/|//[^\n]*", "", open(os.path.join(CSRC, name)).read(), flags=re.S)
    for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\([^)]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i]


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_peers_are_known_to_run_before_their_memory_is_accessed(name):
    for kernel, body in _kernels(name):
        access = ACCESS.search(body)
        if not access:
            continue
        before = body[:access.start()]
        arrive, wait = before.find("cluster_arrive_started"), before.find("cluster_wait_started(")
        whole = before.find("mp_cluster_sync(")              # the dispatch kernel: a whole barrier, on the only path
        assert whole >= 0 or 0 <= arrive < wait, kernel


def test_the_search_finds_the_kernels():
    found = {k for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) for k, b in _kernels(f) if ACCESS.search(b)}
    assert found >= {"exl3_gemv_kernel", "exl3_gemv_tc_kernel", "exl3_gemm_tc_kernel", "moe_dispatch_kernel"}


def test_arrivals_on_a_peers_barrier_release_at_cluster_scope():
    """An arrival on another block's mbarrier publishes what its block wrote: only a release at cluster scope does."""
    remote = []
    for name in sorted(os.listdir(CSRC)):
        text = re.sub(r"/\*.*?\*/|//[^\n]*", "", open(os.path.join(CSRC, name)).read(), flags=re.S)
        remote += re.findall(r"mbarrier\.arrive[\w.:]*\.shared::cluster[\w.]*", text)
    assert remote and all(".release.cluster." in r for r in remote), remote
