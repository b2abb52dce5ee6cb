"""Kernels whose clusters use distributed shared memory: a CTA's shared memory may be accessed only once all
CTAs of the cluster are known to run, so in the source of every kernel a cluster-wide wait comes before
the first access to another CTA's memory, and another one after the last (read from the sources: a race is
not something a run shows)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mdsm_gb300",
                    "csrc")
REMOTE = re.compile(r"map_shared_rank|\bmapa\b|shared::cluster\b(?!\.global)")
WAIT = re.compile(r"\.sync\(\)|barrier_wait\(|barrier\.cluster\.wait")


def _strip(src):
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", src, flags=re.S))


def _kernels():
    """(file, kernel, body) of every kernel that touches another CTA's shared memory."""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        src = _strip(open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__global__", src):
            i = src.index("{", m.start())
            depth, j = 1, i + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[j], 0)
                j += 1
            body = src[i:j]
            if "map_shared_rank" in body or "mapa" in body:
                out.append((f, re.search(r"(k_\w+)\s*\(", src[m.start():i]).group(1), body))
    return out


@pytest.mark.parametrize("f,name,body", _kernels(), ids=lambda v: v if len(v) < 40 else "")
def test_cluster_waits_around_remote_accesses(f, name, body):
    remote = [m.start() for m in REMOTE.finditer(body)]
    waits = [m.start() for m in WAIT.finditer(body) if "cl" in body[max(0, m.start() - 4):m.end()]]
    assert waits, "no cluster-wide wait"
    assert waits[0] < remote[0], "remote access before the cluster's CTAs are known to run"
    assert waits[-1] > remote[-1], "a CTA may exit while another still accesses its memory"
