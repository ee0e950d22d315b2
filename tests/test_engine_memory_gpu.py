"""Device memory comes back when an engine is closed, whatever it was used for."""

import numpy as np
import pytest

from fastlbp_b200 import BatchEngine, CausalFactorGraph, Engine, SetsEngine, api, workloads

pytestmark = pytest.mark.gpu


def _bingo(nt, seed=3):
    fl = workloads.bingo_graph(nt, int(1.5 * nt), max(2, nt // 20), workloads.uniform_int(2, 4),
                               workloads.uniform_int(1, 6), seed, n_alarms=4)
    return CausalFactorGraph.from_factors(fl).graph_arrays()


def _seq(a, state):
    if not state:
        state.append(api.update_seq(a, "SEQFIX", seed=7))
    e = Engine(a)
    e.set_update_seq(state[0])
    e.init()
    e.run_fixed(1)
    return e


def _sets(a, state):
    e = SetsEngine(a, [{k: 1} for k in range(20)])
    e.init()
    e.run_sets_tol(1e-6, 2)
    e.beliefs()
    return e


def _batch(a, state):
    e = BatchEngine([a, a])
    e.init()
    e.run_batch_tol(1e-6, 2)
    e.beliefs()
    return e


def _gradient(a, state):
    e = Engine(a)
    e.adjoint_forward(4, 2)
    e.adjoint_backward(np.ones(e.n_vars))
    return e


@pytest.mark.parametrize("make", [_seq, _sets, _batch, _gradient])
def test_closed_engines_leave_nothing(make):
    import torch

    a, state = _bingo(10_000), []
    for _ in range(5):  # the pool has grown to what one engine needs
        make(a, state).close()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    n = 80
    for _ in range(n):
        make(a, state).close()
    torch.cuda.synchronize()
    lost = free - torch.cuda.mem_get_info()[0]
    assert lost < n * 4 * a["slot_var"].size  # one word an edge slot and engine
