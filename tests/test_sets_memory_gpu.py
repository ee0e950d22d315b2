"""Device memory of an engine of evidence sets beyond the run state: lists of
the clamped entries, and on engines whose sets run on clusters, from their
first run, a bit for every entry of every set.
"""

import pytest

from fastlbp_b200 import CausalFactorGraph, SetsEngine, workloads

pytestmark = pytest.mark.gpu


def _bingo(nt):
    fl = workloads.bingo_graph(nt, int(1.5 * nt), max(2, nt // 20), workloads.uniform_int(2, 4),
                               workloads.uniform_int(1, 6), 3, n_alarms=4)
    return CausalFactorGraph.from_factors(fl).graph_arrays()


@pytest.mark.parametrize("tuples,clusters", [(2000, True), (60_000, False)])
def test_bits_of_cut_entries(tuples, clusters):
    a, n = _bingo(tuples), 100
    e = SetsEngine(a, [{k: k % 2} for k in range(n)])
    none = SetsEngine(a, [{} for _ in range(n)])
    created = e.stats()["bytes"] - none.stats()["bytes"]
    for x in (e, none):
        x.init()
        x.run_sets_tol(1e-6, 3)
    ran = e.stats()["bytes"] - none.stats()["bytes"]
    e.close()
    none.close()
    bits = n * a["slot_var"].size // 8  # a bit for every edge slot of every set; there are somewhat fewer entries
    assert created < bits // 2
    assert (ran - created > bits // 4) == clusters
