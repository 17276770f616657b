"""A plain solver that stops on a bad value or a negative time step: what it
reports and what it leaves, on either side of each size that picks a kernel
(GPU)."""
import numpy as np
import pytest

import mgcfd

pytestmark = pytest.mark.gpu


def _levels(n, nl, seed=3):
    """The levels of a generated mesh, writable."""
    return [mgcfd.Level(**{k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in L.__dict__.items()
                           if k != "owner"}) for L in mgcfd.HostMesh.generate(n, nl, seed).levels()]


# The coarse level of 162^3 (81^3 nodes) is one whose begun state lies in `old` alone.
@pytest.mark.parametrize("form", ["mixed", "dw"])
@pytest.mark.parametrize("n", [40, 162])
def test_restriction_that_finds_bad_values_is_whole(n, form):
    """The restriction that finds a bad level-0 value ends its own launch: every
    level-1 node holds the mean of its children (mg.h:29-64), NaN where a child
    is (the two ends of a bad edge and, after three stages, the nodes within two
    edges of them: at most fifty).  A mean of at most eight terms and the
    reciprocal of their number: within 2^-48 of the value."""
    levels = _levels(n, 2)
    # An inner edge at the start of the solver's node order, so that most of the restriction's blocks follow it.
    e2n, x = levels[0].edge_to_nodes, levels[0].coords
    e = np.argmin(np.abs(0.5 * (x[e2n[:, 0]] + x[e2n[:, 1]]) - 3.0 / n).max(axis=1))
    levels[0].edge_weights[e, :] = np.nan
    s = mgcfd.Solver(levels, 0.5, 3.0, precision=form)
    s.run(2)
    assert s.synchronize() == mgcfd._lib.ERR_BAD_VALUES
    fine, coarse = s.fetch(0), s.fetch(1)
    s.close()
    up = levels[0].node_to_mg
    count = np.bincount(up, minlength=len(coarse))
    assert count.min() > 0
    want = np.stack([np.bincount(up, weights=fine[:, k], minlength=len(coarse)) for k in range(5)], 1) / count[:, None]
    bad = np.isnan(want)
    assert 0 < bad.any(axis=1).sum() <= 50
    assert np.isnan(coarse[bad]).all()
    scale = np.nanmax(np.abs(want), axis=0)
    np.testing.assert_allclose(coarse[~bad], want[~bad], rtol=0, atol=2.0 ** -48 * scale.max())
