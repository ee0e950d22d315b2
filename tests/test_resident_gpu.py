"""Runs of the resident kernel against the pass kernels, bit for bit.

Small graphs run whole on the GPU without further launches; per-pass timing
mode keeps the two launches per sweep. Both evaluate every item by the same
arithmetic, so beliefs, low-pass beliefs, messages, sweep counts and stop
reasons must be equal, from one group of factors up to graphs with items of
every class, for fixed runs (one of them longer than a launch's sweeps),
tolerance and low-pass runs, continued runs, and batches whose graphs share
groups.
"""

import numpy as np
import pytest

from fastlbp_b200 import BatchEngine, CausalFactorGraph, Engine, SetsEngine, workloads
from test_engine_gpu import _large_item_graph
from test_forms_gpu import _with_isolated

pytestmark = pytest.mark.gpu


def _bingo(nt, seed=3, clamps=0):
    fl = workloads.bingo_graph(nt, int(1.5 * nt), max(2, nt // 20), workloads.uniform_int(2, 4),
                               workloads.uniform_int(1, 6), seed, n_alarms=max(1, clamps))
    g = CausalFactorGraph.from_factors(fl)
    if clamps:
        g.clamp_labels({int(a): k % 2 for k, a in enumerate(fl.alarms[:clamps])})
        g = g.rebuild()
    return g.graph_arrays()


def _large():
    g = CausalFactorGraph.from_factors(_with_isolated(_large_item_graph(11)))
    g.clamp_labels({1203: 1, 1207: 0, 5: 1})
    return g.rebuild().graph_arrays()


GRAPHS = {"one_group": lambda: _bingo(12), "two_groups": lambda: _bingo(33), "small": lambda: _bingo(400, clamps=9),
          "zipf": lambda: CausalFactorGraph.from_factors(workloads.config1(5, scale=0.01)).graph_arrays(),
          "large_items": _large}


def _equal(a, b, what):
    assert len(a) == len(b)
    for k, (x, y) in enumerate(zip(a, b)):
        assert np.array_equal(x, y, equal_nan=True), (what, k)


def _runs(e, timed):
    e.set_kernel_timing(timed)
    out = []
    e.reset_counts()
    e.init()
    e.run_fixed(7)
    e.run_fixed(1)  # a continued run
    out += [e.beliefs(), *e.fv_messages(), *e.vf_messages()]
    e.reset_counts()
    e.init()
    info = e.run_tol(1e-6, 60, 1e9)
    again = e.run_tol(1e-9, 70, 1e9)
    out += [e.beliefs(), [info[k] for k in ("sweeps", "reason", "maxdiff")], [again[k] for k in ("sweeps", "reason")]]
    e.reset_counts()
    e.init()
    info = e.run_lowpass(1e-6, 5, 30, 4)
    out += [e.beliefs(), e.lowpass(), [info[k] for k in ("sweeps", "reason", "frac", "maxdiff")], *e.fv_messages()]
    e.set_kernel_timing(False)
    return out


@pytest.mark.parametrize("graph", sorted(GRAPHS))
@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("damping", [0.0, 0.2])
def test_resident_equals_passes(graph, prec, damping):
    e = Engine(GRAPHS[graph](), precision=prec, damping=damping)
    _equal(_runs(e, False), _runs(e, True), graph)
    e.close()


def test_run_longer_than_a_launch():
    e = Engine(_bingo(30), damping=0.1)
    got = []
    for timed in (False, True):
        e.set_kernel_timing(timed)
        e.init()
        e.run_fixed(4096 + 5)
        got.append([e.beliefs(), *e.vf_messages()])
    _equal(got[0], got[1], "long")
    e.close()


def test_more_variables_than_cached_rows():
    """Enough variables without entries that a block's items exceed its table of cached constants."""
    a = dict(_bingo(300))
    a["n_vars"] = 6_000_000
    e = Engine(a)
    _equal(_runs(e, False), _runs(e, True), "rows")
    e.close()


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("damping", [0.0, 0.1])
def test_batch_equals_passes(prec, damping):
    graphs = [_bingo(n, seed=n, clamps=n % 7) for n in (13, 40, 9, 700, 75, 2100, 31)] + [_large()]
    e = BatchEngine(graphs, precision=prec, damping=damping)
    got = []
    for timed in (False, True):
        e.set_kernel_timing(timed)
        e.reset_counts()
        e.init()
        one = e.run_batch_tol(1e-6, 25)
        got.append([e.beliefs(), *one, *e.fv_messages(), *e.vf_messages()])
    _equal(got[0], got[1], "batch")
    e.close()


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("damping", [0.0, 0.2])
def test_sets_equal_passes(prec, damping):
    """Evidence sets taken by clusters (7 jobs of one graph, cut entries of large
    variables among them) against the two-launch form."""
    fl = workloads.config1(8, scale=0.003)
    a = CausalFactorGraph.from_factors(fl).graph_arrays()
    deg = np.bincount(a["slot_var"], minlength=a["n_vars"])
    vs = np.argsort(-deg)[:12]
    sets = [{int(v): int(v + k) % 2 for v in vs[:2 * k]} for k in range(7)]
    got = []
    for timed in (False, True):
        e = SetsEngine(a, sets, precision=prec, damping=damping)
        e.set_kernel_timing(timed)
        e.init()
        one = e.run_sets_tol(1e-6, 40)
        got.append([e.beliefs(), *one])
        e.close()
    _equal(got[0], got[1], "sets")


def test_batch_continued_and_limited():
    """A second call continues from the first one's messages; a sweep limit ends some graphs."""
    graphs = [_bingo(n, seed=n) for n in (20, 800, 90)]
    e = BatchEngine(graphs, damping=0.1)
    got = []
    for timed in (False, True):
        e.set_kernel_timing(timed)
        e.reset_counts()
        e.init()
        one = e.run_batch_tol(1e-6, 9)
        two = e.run_batch_tol(1e-5, 30)
        info = e.info.as_dict()
        got.append([*one, *two, e.beliefs(), [info["sweeps"], info["reason"], info["maxdiff"]], *e.vf_messages()])
    _equal(got[0], got[1], "continued")
    e.close()


@pytest.mark.parametrize("prec", [32, 64])
def test_batch_out_of_time(prec):
    """No time at all: one sweep of every graph, the ones too large for a cluster too."""
    graphs = [_bingo(n, seed=n) for n in (20, 300, 90)] + [_large()]
    e = BatchEngine(graphs, precision=prec)
    got = []
    for timed in (False, True):
        e.set_kernel_timing(timed)
        e.reset_counts()
        e.init()
        sweeps, reasons = e.run_batch_tol(1e-9, 30, 1e-9)
        assert np.all(np.asarray(sweeps) == 1)
        got.append([e.beliefs(), reasons, [e.info.as_dict()["reason"]], *e.vf_messages()])
    _equal(got[0], got[1], "out of time")
    e.close()


def test_batch_time_over_several_launches():
    """The time limit counts from the call, not from a launch of 4,096 sweeps."""
    e = BatchEngine([_bingo(n, seed=n) for n in (20, 90)])
    sweeps, _ = e.run_batch_tol(-1.0, 400_000, 0.1)  # no belief is ever settled
    assert np.all((np.asarray(sweeps) > 4096) & (np.asarray(sweeps) < 400_000))
    e.close()
