"""FP64 forms in combinations that pick their own code: small levels under every
numbering and set-up, and the whole-row increments at every block size (GPU)."""
import numpy as np
import pytest

import mgcfd
from irregular import irregular_levels
from test_gpu_variants import _small_levels

pytestmark = pytest.mark.gpu


def _solve(levels, **opts):
    s = mgcfd.Solver(levels, 0.55, 2.5, **opts)
    s.run(2)
    assert s.synchronize() == 0
    out = [s.fetch(l) for l in range(len(levels))], s.norms()[1:]
    s.close()
    return out


def _same(a, b):
    """The same sums in another order: a few 1e-16 of the state; norms as test_gpu_variants.py derives."""
    for x, y in zip(a[0], b[0]):
        np.testing.assert_allclose(x, y, rtol=0, atol=1e-13 * np.abs(y).max())
    np.testing.assert_allclose(a[1], b[1], rtol=1e-6, atol=0)


@pytest.mark.parametrize("renumber,host_setup", [("spatial", True), ("none", False), ("none", True), ("rcm", True)])
@pytest.mark.parametrize("kind", ["3", "8", "16", "irregular", "hub"])
def test_small_levels_under_every_numbering_and_setup(kind, renumber, host_setup):
    """k_stage_small in FP64 (no increment named), its sliced lists built from the
    host's tables and from the device's, against the atomic increment."""
    levels = _small_levels(kind)
    opts = dict(renumber=renumber, host_setup=host_setup)
    _same(_solve(levels, **opts), _solve(levels, increment="atomic", **opts))


@pytest.mark.parametrize("block_size", [32, 256, 1024])
@pytest.mark.parametrize("kind", ["lattice", "irregular"])
def test_whole_row_increments_at_every_block_size(kind, block_size):
    """k_flux_f64's atomics pass through shared memory sized by the block; edge
    counts that leave a ragged last warp, and warps without an edge."""
    levels = mgcfd.HostMesh.generate(9, 2, 5).levels() if kind == "lattice" else irregular_levels(700, 2, 4)
    assert levels[0].nedges % 32 and levels[1].nedges % 32
    _same(_solve(levels, increment="atomic", block_size=block_size), _solve(levels, increment="gather"))
