"""CPU: no cluster kernel touches another CTA's shared memory before a cluster
barrier has shown that every CTA of the cluster has started (distributed shared
memory does not exist before), nor lets a CTA leave while its words may still be
read.  Read from the source: whether a missing barrier shows on a device depends
on timing, and a lost access can fault."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cuda-moea_b200" / "csrc"
REMOTE = re.compile(r"\bmap_shared_rank\s*\(|\bgrp\.map\s*\(")
BARRIER = re.compile(r"\b(?:cluster|grp|g)\.sync\s*\(\s*\)")


def _bodies(text):
    """(name, body, text before) of everything that looks like a function."""
    text = re.sub(r"//[^\n]*", "", text)
    text = re.sub(r"__(?:cluster_dims|launch_bounds)__\s*\([^()]*\)", "", text)
    for m in re.finditer(r"\b(\w+)\s*\([^;{}]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i], text[max(0, m.start() - 200):m.start()]


def _kernels():
    found = []
    for path in sorted(CSRC.glob("*.cu*")):
        for name, body, before in _bodies(path.read_text()):
            kernel = "__global__" in before[max(before.rfind("}"), before.rfind(";"), 0):]
            if REMOTE.search(body) and (kernel or name == "niche_buckets"):
                found.append((path.name, name, body))
    return found


def test_the_kernels_are_found():
    assert {"dir_delta_kernel", "ideal_kernel", "nsga3_prep", "nds_fronts", "niche_buckets"} <= {k[1] for k in _kernels()}


@pytest.mark.parametrize("name,body", [pytest.param(k[1], k[2], id=f"{k[0]}:{k[1]}") for k in _kernels()])
def test_first_remote_access_follows_a_barrier(name, body):
    first = REMOTE.search(body).start()
    assert BARRIER.search(body[:first]), f"{name}: remote shared memory before any cluster barrier"


@pytest.mark.parametrize("name,body", [pytest.param(k[1], k[2], id=f"{k[0]}:{k[1]}") for k in _kernels()])
def test_a_barrier_follows_the_last_remote_access(name, body):
    last = [m.end() for m in REMOTE.finditer(body)][-1]
    assert BARRIER.search(body[last:]), f"{name}: a CTA may leave while its shared memory is read"
