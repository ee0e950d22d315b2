"""Which form a run takes: whole runs in one launch where that is the faster
form, two passes a sweep elsewhere, counted by the launches a run reports; and
the same results either way (per-pass timing mode forces the passes).
"""

import numpy as np
import pytest

from fastlbp_b200 import BatchEngine, CausalFactorGraph, Engine, SetsEngine, workloads

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


def _batch(graphs, prec, sweeps, passes=False):
    e = BatchEngine(graphs, precision=prec)
    e.set_kernel_timing(passes)
    e.init()
    stops = e.run_batch_tol(1e-6, sweeps)
    info = e.info.as_dict()
    out = [e.beliefs(), *stops, [info[k] for k in ("sweeps", "reason", "maxdiff")], *e.vf_messages()]
    e.close()
    return info, out


# batches on clusters or resident, on clusters with the rest in the passes, and all in the passes
@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("sizes,one_launch", [
    ([300] * 5 + [1000] * 3, True), ([9000, 9100, 9200], True),
    ([1000 + k for k in range(24)] + [70_000, 71_000], False), ([60_000, 61_000, 62_000], False),
], ids=["small", "resident", "both", "passes"])
def test_batches(prec, sizes, one_launch):
    graphs = [_bingo(n, seed=k + 1) for k, n in enumerate(sizes)]
    info, got = _batch(graphs, prec, 25)
    _, want = _batch(graphs, prec, 25, passes=True)
    assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(got, want))
    assert (info["launches"] == 1) == one_launch


def test_thousands_of_tiny_graphs():
    """More graphs than clusters take in a reasonable number of rounds, and than the resident kernel counts."""
    kinds = [_bingo(60 + k, seed=k + 1) for k in range(7)]
    info, got = _batch(kinds * 800, 32, 40)
    assert info["launches"] > 1
    n = sum(a["n_vars"] for a in kinds)
    alone, sweeps = [], []
    for a in kinds:
        e = Engine(a)
        e.init()
        sweeps.append(e.run_tol(1e-6, 40, 1e9)["sweeps"])
        alone.append(e.beliefs())
        e.close()
    for at in (0, 399, 799):
        assert np.array_equal(got[0][at * n:(at + 1) * n], np.concatenate(alone))
    assert list(got[1]) == sweeps * 800


@pytest.mark.parametrize("tuples,n_sets,one_launch", [(2000, 1, True), (20_000, 1, False), (20_000, 3, True)])
def test_evidence_sets(tuples, n_sets, one_launch):
    sets = [{3: 1, 10 + k: k % 2} for k in range(n_sets)]
    got = []
    for passes in (False, True):
        e = SetsEngine(_bingo(tuples), sets)
        e.set_kernel_timing(passes)
        e.init()
        stops = e.run_sets_tol(1e-6, 25)
        got.append([e.beliefs(), *stops])
        if not passes:
            assert (e.info.as_dict()["launches"] == 1) == one_launch
        e.close()
    assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(*got))
