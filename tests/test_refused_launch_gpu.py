"""A launch of a whole run that CUDA refuses (a context limited to part of the
SMs, for instance) leaves the run to the pass kernels, with the same results.
The refusal is an error code returned in place of the launch.
"""

import numpy as np
import pytest

from fastlbp_b200 import BatchEngine, CausalFactorGraph, Engine, SetsEngine, _native, workloads

pytestmark = pytest.mark.gpu

TUPLES = {"cluster": 200, "resident": 8000}


def _bingo(nt, seed=3):
    fl = workloads.bingo_graph(nt, int(1.5 * nt), max(2, nt // 20), workloads.uniform_int(2, 4),
                               workloads.uniform_int(1, 6), seed, n_alarms=4)
    return CausalFactorGraph.from_factors(fl).graph_arrays()


def _refuse(e, n):
    _native.check(_native.lib().flbp_test_refuse_launches(e._h, n))


def _fixed(e):
    e.run_fixed(9)
    return [e.beliefs(), *e.vf_messages()]


def _long(e):  # two launches
    e.run_fixed(4096 + 3)
    return [e.beliefs(), *e.vf_messages()]


def _tol(e):
    info = e.run_tol(1e-6, 40, 1e9)
    return [e.beliefs(), [info[k] for k in ("sweeps", "reason", "maxdiff")], *e.vf_messages()]


def _lowpass(e):
    info = e.run_lowpass(1e-6, 5, 30, 4)
    return [e.beliefs(), e.lowpass(), [info[k] for k in ("sweeps", "reason", "frac", "maxdiff")]]


def _gradient(e):
    out = [e.adjoint_forward(11, 4)]
    return out + list(e.adjoint_backward(np.linspace(-1.0, 1.0, e.n_vars)))


def _equal(a, b):
    assert len(a) == len(b)
    assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))


@pytest.mark.parametrize("size", sorted(TUPLES))
@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("run", [_fixed, _long, _tol, _lowpass, _gradient])
@pytest.mark.parametrize("n", [1, 2])
def test_refused_run(size, prec, run, n):
    """n = 1: the first kind of launch only; 2: of a small graph both kinds."""
    a = _bingo(TUPLES[size] if run is not _long else TUPLES[size] // 10)
    got = []
    for refused in (0, n):
        e = Engine(a, precision=prec)
        e.init()
        _refuse(e, refused)
        got.append(run(e))
        e.close()
    _equal(got[0], got[1])


@pytest.mark.parametrize("n", [1, 2])
def test_refused_batch_and_sets(n):
    graphs = [_bingo(k, seed=k) for k in (20, 90, 300)]
    sets = [{0: 1}, {1: 0, 2: 1}, {}]
    for make, run in ((lambda: BatchEngine(graphs), lambda e: e.run_batch_tol(1e-6, 40)),
                      (lambda: SetsEngine(graphs[2], sets), lambda e: e.run_sets_tol(1e-6, 40))):
        got = []
        for refused in (0, n):
            e = make()
            e.init()
            _refuse(e, refused)
            one = run(e)
            info = e.info.as_dict()
            got.append([*one, e.beliefs(), [info[k] for k in ("sweeps", "reason", "maxdiff")]])
            e.close()
        _equal(got[0], got[1])
