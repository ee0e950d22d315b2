"""Blocks of a cluster are scheduled together but do not start at the same
instant: a kernel may store to another block's shared memory only after a
cluster barrier that follows its entry. Read from the kernel's source, since a
launch that broke the rule could fault the GPU; then many short launches of
the kernel, whose first remote store is the one at risk.
"""

import os
import re

import numpy as np
import pytest

import fastlbp_b200
from fastlbp_b200 import CausalFactorGraph, Engine, workloads

CSRC = os.path.join(os.path.dirname(os.path.abspath(fastlbp_b200.__file__)), "csrc")


def _kernels(text):
    """(name, body without comments) of every __global__ function."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    for m in re.finditer(r"__global__", text):
        head = text[m.start():text.index("{", m.start())]
        depth, end = 0, m.start() + len(head)
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        yield re.findall(r"(\w+)\s*\(", head)[-1], text[m.start() + len(head):end]


def test_barrier_before_the_first_remote_store():
    seen = 0
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, f)) as fh:
            text = fh.read()
        if "shared::cluster" not in text:
            continue
        for name, body in _kernels(text):
            store = re.search(r"\bcluster_st\(", body)
            if store:
                seen += 1
                barrier = re.search(r"\bcluster_sync_all\(\)", body)
                assert barrier and barrier.start() < store.start(), (f, name)
    assert seen


@pytest.mark.gpu
@pytest.mark.parametrize("tuples", [12, 400, 3000])
def test_many_short_launches(tuples):
    fl = workloads.bingo_graph(tuples, int(1.5 * tuples), max(2, tuples // 20), workloads.uniform_int(2, 4),
                               workloads.uniform_int(1, 6), 3, n_alarms=1)
    e = Engine(CausalFactorGraph.from_factors(fl).graph_arrays())
    e.set_kernel_timing(True)  # two launches a sweep
    e.init()
    e.run_fixed(1)
    want = e.beliefs()
    e.set_kernel_timing(False)
    for _ in range(300):
        e.init()
        e.run_fixed(1)
        assert np.array_equal(e.beliefs(), want)
    e.close()
