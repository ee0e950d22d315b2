"""Gradients whose sweeps run in one launch a segment against two launches a
sweep, bit for bit.

Per-pass timing mode forces the two launches, which graphs above a million
slots take by themselves. Checkpoint intervals of one sweep, intervals that do
not divide the sweeps, and segments of more sweeps than one launch makes.
"""

import numpy as np
import pytest

from fastlbp_b200 import BatchEngine, CausalFactorGraph, Engine, workloads
from test_engine_gpu import _large_item_graph

pytestmark = pytest.mark.gpu


def _bingo(nt, seed=3):
    fl = workloads.bingo_graph(nt, int(1.5 * nt), max(2, nt // 20), workloads.uniform_int(2, 4),
                               workloads.uniform_int(1, 6), seed, n_alarms=4)
    return CausalFactorGraph.from_factors(fl).graph_arrays()


def _large():
    return CausalFactorGraph.from_factors(_large_item_graph(11)).graph_arrays()


MAKE = {"small": lambda p: Engine(_bingo(300), precision=p), "large_items": lambda p: Engine(_large(), precision=p),
        "batch": lambda p: BatchEngine([_bingo(n, seed=n) for n in (40, 700, 9)], precision=p)}


def _equal_forms(e, sweeps, every):
    grad = np.random.default_rng(5).normal(size=e.n_vars)
    got = []
    for passes in (False, True):
        e.set_kernel_timing(passes)
        before = e.stats()["launches"]
        b = e.adjoint_forward(sweeps, every)
        forward = e.stats()["launches"] - before
        got.append([b, *e.adjoint_backward(grad), *e.vf_messages()])
        # either a launch or two a segment, or two a sweep; and the beliefs
        assert (forward > sweeps) == passes or sweeps < 3 or every < 3
    e.close()
    for x, y in zip(*got):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("graph", sorted(MAKE))
@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("sweeps,every", [(1, 1), (5, 1), (11, 4), (12, 4), (7, 20)])
def test_resident_segments_equal_passes(graph, prec, sweeps, every):
    _equal_forms(MAKE[graph](prec), sweeps, every)


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("sweeps,every", [(4096 + 3, 5000), (4096 + 3, 4096 + 1)])
def test_segment_longer_than_a_launch(prec, sweeps, every):
    _equal_forms(Engine(_bingo(12), precision=prec), sweeps, every)
