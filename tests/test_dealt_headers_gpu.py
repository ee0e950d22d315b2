"""Tile counts at the edges of the staged factor pass's dealt headers.

A block reads the headers of its tiles 32 at a time from a row of equal
length for every block, empty headers behind its last tile: one tile for the
whole grid, one more tile than blocks, and more than 32 tiles a block. The
direct forms use no tiles; both give the same bits.
"""

import numpy as np
import pytest

from fastlbp_b200 import Engine

pytestmark = pytest.mark.gpu

TILE = 512  # one-body factors of a tile
BLOCKS = 2 * 148


def _chain(n):
    """n AND factors x_i -> x_(i+1) and a prior on every variable."""
    rng = np.random.default_rng(n)
    v = np.arange(n + 1)
    slots = np.concatenate([np.stack([v[:-1], v[1:]], 1).ravel(), v])
    off = np.concatenate([2 * np.arange(n), 2 * n + np.arange(n + 2)])
    return dict(n_vars=n + 1, factor_offsets=off, slot_var=slots,
                factor_head=np.concatenate([2 * np.arange(n) + 1, 2 * n + v]),
                factor_type=np.concatenate([np.ones(n, np.int32), np.zeros(n + 1, np.int32)]),
                factor_p=rng.uniform(0.6, 0.95, 2 * n + 1),
                factor_q=np.concatenate([rng.uniform(0.0, 0.3, n), np.zeros(n + 1)]))


@pytest.mark.parametrize("n", [1, TILE * BLOCKS + 1, TILE * BLOCKS * 33 + 1])
def test_staged_equals_direct(n):
    e = Engine(_chain(n))
    got = []
    for forms in ((0, 0), (1, 1)):
        e.set_tuning(*forms)
        e.set_kernel_timing(True)  # two passes per sweep
        e.reset_counts()
        e.init()
        e.run_fixed(5)
        got.append(e.beliefs())
    assert np.array_equal(got[0], got[1])
    assert np.all((got[0] > 0.0) & (got[0] < 1.0))
