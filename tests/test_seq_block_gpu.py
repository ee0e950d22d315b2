"""The one-block form of a sequential sweep against two launches per batch, bit for bit.

The block evaluates four factors of up to eight body slots per warp and wider
ones a warp each; the two-launch form takes a warp per factor throughout.
Fan-ins at the edges of the packed and the one-warp widths, clamped heads,
item counts that leave groups of four unfilled, and a batch whose staged
outputs exceed the block's shared memory.
"""

import numpy as np
import pytest

from fastlbp_b200 import CausalFactorGraph, Engine, SetsEngine, api, workloads

pytestmark = pytest.mark.gpu


def _mixed(n, fans, seed=4):
    """n factors over random inputs, fan-ins in turn from `fans`, AND and OR alternating."""
    rng = np.random.default_rng(seed)
    kind, head, off, body, p, q = [], [], [0], [], [], []
    for i in range(n):
        k = fans[i % len(fans)]
        kind.append(workloads.AND if i % 2 else workloads.OR)
        head.append(10_000 + i)
        body += [int(x) for x in rng.choice(400 + i, size=k, replace=False)]
        off.append(len(body))
        p.append(0.9 if i % 2 else 1.0)
        q.append(0.05 if i % 3 == 0 else 0.0)
    fl = workloads.FactorList(np.array(kind, np.int32), np.array(head, np.int64), np.array(off, np.int64),
                              np.array(body, np.int64), np.array(p), np.array(q))
    used = np.unique(fl.body)
    m = used.size
    return workloads.FactorList(np.concatenate([fl.kind, np.zeros(m, np.int32)]), np.concatenate([fl.head, used]),
                                np.concatenate([fl.body_off, np.full(m, fl.body_off[-1])]), fl.body,
                                np.concatenate([fl.p, rng.uniform(0.2, 0.8, m)]), np.concatenate([fl.q, np.zeros(m)]))


def _beliefs(a, upd, prec, damping, sweeps):
    e = Engine(a, precision=prec, damping=damping)
    e.set_update_seq(api.update_seq(a, upd, seed=7))
    out = []
    for kernel in (1, 2):
        e.set_seq_kernel(kernel)
        e.init()
        e.run_fixed(sweeps)
        out.append(e.beliefs())
        out.append(e.fv_messages())
    e.close()
    return out


@pytest.mark.parametrize("fans", [(1, 2, 3), (7, 8, 9), (8,), (31, 32, 33, 2), (257, 3, 300, 8, 1)])
@pytest.mark.parametrize("prec,damping", [(32, 0.0), (64, 0.0), (32, 0.2)])
@pytest.mark.parametrize("upd", ["SEQFIX", "TOPO"])
def test_block_equals_launches(fans, prec, damping, upd):
    g = CausalFactorGraph.from_factors(_mixed(61, fans))
    g.clamp_labels({10_003: 1, 10_008: 0, 5: 1, 17: 0})
    b1, m1, b2, m2 = _beliefs(g.rebuild().graph_arrays(), upd, prec, damping, 4)
    assert np.array_equal(b1, b2, equal_nan=True)
    for x, y in zip(m1, m2):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("prec", [32, 64])
def test_batch_larger_than_shared_staging(prec):
    """30,000 separate factors: one batch of 120,000 staged messages."""
    n = 30_000
    ids = np.arange(n, dtype=np.int64)
    fl = workloads.FactorList(np.full(n, workloads.AND, np.int32), 4 * ids, 3 * np.arange(n + 1, dtype=np.int64),
                              np.stack([4 * ids + 1, 4 * ids + 2, 4 * ids + 3], 1).ravel(),
                              np.full(n, 0.9), np.full(n, 0.1))
    b1, m1, b2, m2 = _beliefs(CausalFactorGraph.from_factors(fl).graph_arrays(), "SEQFIX", prec, 0.0, 2)
    assert np.array_equal(b1, b2) and all(np.array_equal(x, y) for x, y in zip(m1, m2))


def test_set_beliefs_read_in_several_pieces():
    """More values than one gather takes: every set's row in its place."""
    fl = workloads.config0(3)
    a = dict(CausalFactorGraph.from_factors(fl).graph_arrays())
    n = a["n_vars"]
    a["n_vars"] = 300_000
    sets = [{int(5 * k): k % 2} for k in range(40)]
    e = SetsEngine(a, sets)
    e.init()
    e.run_sets_tol(1e-6, 3)
    b = e.beliefs()
    e.close()
    assert b.shape == (40, 300_000) and np.all(b[:, n:] == 0.5)
    for k in (0, 1, 26, 27, 28, 39):
        s = SetsEngine(a, [sets[k]])
        s.init()
        s.run_sets_tol(1e-6, 3)
        assert np.array_equal(s.beliefs()[0], b[k], equal_nan=True), k
        s.close()
