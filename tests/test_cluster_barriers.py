"""Distributed shared memory may be touched only once every block of the cluster
runs, which nothing but a barrier of the cluster tells.  A kernel that lacks it
works as long as all blocks start in time, so no run shows the fault: the source
is read instead.  Every kernel that maps another block's shared memory has a
barrier of the whole cluster before the first such access, and one behind the
last (a block must not leave while others may still reach into it)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "chemrust-scf_b200", "csrc")
BARRIER = re.compile(r"(this_cluster\(\)|\bcluster|\bcl)\s*\.\s*sync\(\)|barrier\.cluster\.wait")
REMOTE = re.compile(r"map_shared_rank|\bmapa\b")


def _kernels(text):
    """(name, body) of every __global__ function that is defined in text."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    for m in re.finditer(r"__global__", text):
        start = text.index("{", m.end())
        head = text[m.end():start]
        if ";" in head:
            continue
        depth, at = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
            if depth == 0:
                break
        head = re.sub(r"__\w+__\s*\((?:[^()]|\([^()]*\))*\)", "", head)
        yield re.search(r"(\w+)\s*\(", head).group(1), text[start:at]


def _cluster_kernels():
    out = []
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as h:
                out += [(f, name, body) for name, body in _kernels(h.read()) if REMOTE.search(body)]
    return out


@pytest.mark.parametrize("where,name,body", _cluster_kernels(),
                         ids=lambda v: v if len(v) < 40 else "")
def test_barriers_around_remote_accesses(where, name, body):
    first = REMOTE.search(body).start()
    last = [m.start() for m in REMOTE.finditer(body)][-1]
    at = [m.start() for m in BARRIER.finditer(body)]
    assert any(b < first for b in at), "%s %s: remote access before any cluster barrier" % (where, name)
    assert any(b > last for b in at), "%s %s: no cluster barrier behind the last access" % (where, name)


def test_kernels_are_found():
    assert {"k_minmax", "k_tridiag"} <= {name for _, name, _ in _cluster_kernels()}
