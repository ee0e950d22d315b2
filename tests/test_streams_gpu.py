"""An engine's calls use its own stream only: they neither wait for work queued
on the process's default stream nor hold it up.

The default stream is kept busy by a kernel of one thread that ends by itself;
every kind of run has to return while that kernel is still going.
"""

import numpy as np
import pytest

from fastlbp_b200 import BatchEngine, CausalFactorGraph, Engine, SetsEngine, workloads

pytestmark = pytest.mark.gpu


def _bingo(nt, seed=3):
    fl = workloads.bingo_graph(nt, int(1.5 * nt), max(2, nt // 20), workloads.uniform_int(2, 4),
                               workloads.uniform_int(1, 6), seed, n_alarms=4)
    return CausalFactorGraph.from_factors(fl).graph_arrays()


def _batch():
    e = BatchEngine([_bingo(n, seed=n) for n in (20, 90, 300)])

    def run():
        e.init()
        e.run_batch_tol(1e-6, 40)
        return e.beliefs()
    return e, run


def _sets():
    a = _bingo(200)
    e = SetsEngine(a, [{0: 1}, {1: 0, 2: 1}, {}])

    def run():
        e.init()
        e.run_sets_tol(1e-6, 40)
        return e.beliefs()
    return e, run


def _single(nt):
    e = Engine(_bingo(nt))

    def run():
        e.reset_counts()  # the sweep limit counts from here
        e.init()
        e.run_tol(1e-6, 40, 1e9)
        return e.beliefs()
    return e, run


@pytest.mark.parametrize("make", [_batch, _sets, lambda: _single(200), lambda: _single(8000)],
                         ids=["batch", "sets", "small", "resident"])
def test_runs_beside_a_busy_default_stream(make):
    import torch

    e, run = make()
    want = run()  # plans and buffers are made by the first run
    run()
    done = torch.cuda.Event()
    torch.cuda._sleep(1_000_000_000)  # about half a second
    done.record()
    got = run()
    busy = not done.query()
    torch.cuda.synchronize()
    e.close()
    assert np.array_equal(got, want)
    assert busy
