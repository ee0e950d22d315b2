"""Which form a run takes: whole runs in one launch where that is the faster
form, two passes a sweep elsewhere, counted by the launches a run reports; and
the same results either way (per-pass timing mode forces the passes).
"""

import numpy as np
import pytest

from fastlbp_b200 import CausalFactorGraph, Engine, workloads

pytestmark = pytest.mark.gpu

SWEEPS = 12


def _bingo(nt, seed=3):
    fl = workloads.bingo_graph(nt, int(1.5 * nt), max(2, nt // 20), workloads.uniform_int(2, 4),
                               workloads.uniform_int(1, 6), seed, n_alarms=4)
    return dict(CausalFactorGraph.from_factors(fl).graph_arrays())


def _run(e, mode):
    e.reset_counts()
    e.init()
    if mode == "fixed":
        info = e.run_fixed(SWEEPS)
    elif mode == "tol":
        info = e.run_tol(-1.0, SWEEPS, 1e9)
    else:
        info = e.run_lowpass(-1.0, SWEEPS - 2, SWEEPS - 1, 3)
    return info, [e.beliefs(), *([e.lowpass()] if mode == "lowpass" else []), *e.vf_messages()]


def _check(a, prec, mode, one_launch, damping=0.0):
    e = Engine(a, precision=prec, damping=damping)
    info, got = _run(e, mode)
    e.set_kernel_timing(True)
    _, want = _run(e, mode)
    e.close()
    assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(got, want))
    assert (info["launches"] < SWEEPS) == one_launch


# variables without entries beside a graph of 21 k slots
@pytest.mark.parametrize("prec,mode,bare,one_launch", [
    (32, "fixed", 30_000, True), (32, "fixed", 500_000, True), (32, "fixed", 1_000_000, False),
    (32, "tol", 1_000_000, True), (32, "tol", 3_000_000, False),
    (32, "lowpass", 3_000_000, True), (32, "lowpass", 5_000_000, False),
    (64, "fixed", 1_000_000, False), (64, "tol", 3_000_000, False),
    (64, "lowpass", 3_000_000, True),  # more items than a block's table of constants holds
])
def test_variables_without_entries(prec, mode, bare, one_launch):
    a = _bingo(2500)
    a["n_vars"] += bare
    _check(a, prec, mode, one_launch)


# graphs of 708 k and 590 k slots, 12 % of them in factors that take a warp each
@pytest.mark.parametrize("tuples,prec,damping,mode,one_launch", [
    (120_000, 32, 0.0, "fixed", False), (100_000, 32, 0.0, "fixed", True), (100_000, 32, 0.1, "fixed", False),
    (100_000, 64, 0.0, "fixed", False), (100_000, 64, 0.1, "tol", True), (50_000, 64, 0.1, "fixed", True),
])
def test_factors_that_take_a_warp(tuples, prec, damping, mode, one_launch):
    a = CausalFactorGraph.from_factors(workloads.config1(1, scale=tuples / 1_000_000)).graph_arrays()
    _check(a, prec, mode, one_launch, damping)
