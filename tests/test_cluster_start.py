"""Kernels that reach a peer CTA's shared memory, read as source.

A CTA of a cluster may touch another's shared memory only once every CTA of the
cluster has started, which a cluster barrier alone tells.  A kernel that omits
it may lose a store or fault, and only when a CTA starts late, so no run shows
it: the order of the barrier and the accesses is checked in the source instead.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "maos_b200", "csrc")
# data accesses (an address mapped by mapa alone touches nothing)
ACCESS = re.compile(r"\b(dsm_st|dsm_ld|dsm_ld_f64|dsm_peer_f64)\s*\(|(ld|st|red|atom)\.[\w.]*shared::cluster")
WAIT = re.compile(r"\b(cluster_sync_all|cluster_wait|cl_wait)\s*\(|barrier\.cluster\.wait")
ARRIVE = re.compile(r"\b(cluster_sync_all|cluster_arrive\w*|cl_arrive)\s*\(|barrier\.cluster\.arrive")


def _kernels():
    """(name, body) of every __global__ function that reaches a peer's shared memory."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for g in re.finditer(r"__global__", text):
            at = text.index("{", g.start())
            depth, end = 1, at + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            name = re.search(r"(\w+)\s*\([^()]*(\([^()]*\)[^()]*)*\)\s*$", text[g.start():at].rstrip()).group(1)
            body = text[at:end]
            if ACCESS.search(body):
                found.append((name, body))
    return found


def test_the_cluster_kernels_are_found():
    assert {"k_fd_fused", "k_fd_inv", "k_cg_step", "k_gsplit8"} <= {n for n, _ in _kernels()}


@pytest.mark.parametrize("name,body", _kernels(), ids=[n for n, _ in _kernels()])
def test_peers_have_started_before_their_memory_is_touched(name, body):
    first = ACCESS.search(body).start()
    wait = WAIT.search(body)
    assert wait and wait.start() < first, f"{name}: a peer's shared memory is accessed before a cluster barrier"
    # every barrier phase is one arrival and one wait, up to the first access and in all
    assert len(ARRIVE.findall(body[:first])) == len(WAIT.findall(body[:first]))
    assert len(ARRIVE.findall(body)) == len(WAIT.findall(body))
