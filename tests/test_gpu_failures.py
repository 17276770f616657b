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


def _norm_kernel_sizes():
    """Level-0 sizes on either side of the lines that pick the kernel which counts
    bad values: FP64 k_stage_small, k_update; the others k_restrict_small and (a
    coarse level above 16384 nodes) k_restrict."""
    return [("fp64", 8), ("fp64", 20), ("fp64", 40), ("mixed", 8), ("mixed", 40), ("mixed", 64), ("dw", 8), ("dw", 40),
            ("dw", 64)]


@pytest.mark.parametrize("increment", ["auto", "gather"])
@pytest.mark.parametrize("form,n", _norm_kernel_sizes())
def test_bad_values_are_reported_by_every_counting_kernel(form, n, increment):
    levels = _levels(n, 2)
    levels[0].edge_weights[n, :] = np.nan
    s = mgcfd.Solver(levels, 0.5, 3.0, precision=form, increment=increment)
    s.run(2)
    assert s.synchronize() == mgcfd._lib.ERR_BAD_VALUES
    assert "Bad variable values" in mgcfd._lib.load().mgcfd_last_error().decode()
    with pytest.raises(mgcfd._lib.MgcfdError):
        s.run(1)
    s.reset()
    s.run(1)
    assert s.synchronize() == mgcfd._lib.ERR_BAD_VALUES  # a reset solver finds them again
    s.close()


# Level-1 sizes on either side of the lines of k_stage_small (4096, 8192 and 16384 nodes; FP64
# in meshes up to 32768 nodes), and one whose begun state lies in `old` alone (81^3).
@pytest.mark.parametrize("form,n", [("fp64", 16), ("fp64", 32), ("fp64", 36), ("mixed", 16), ("mixed", 54), ("mixed", 162),
                                    ("dw", 16), ("dw", 44), ("dw", 162)])
def test_negative_time_step_stops_every_stage_kernel(form, n):
    """A negative volume on level 1 gives min_dt < 0 there (euler3d.cpp:480-484): the
    solver stops before that level's first stage, so it holds the restricted
    state, as it does with the gather increment (mixed: the same bits; FP64 and
    DW sum level 0 in another order: 2^-40 of each variable's scale)."""
    levels = _levels(n, 2)
    s = mgcfd.Solver(levels, 0.5, 3.0, precision="mixed")
    for l, L in enumerate(levels):
        L.volumes = s.fetch(l, mgcfd.Q_VOLUMES)
    s.close()
    levels[1].volumes[5] *= -1.0
    got = []
    for increment in ("auto", "gather"):
        s = mgcfd.Solver(levels, 0.5, 3.0, precision=form, increment=increment)
        s.run(2)
        assert s.synchronize() == mgcfd._lib.ERR_NEGATIVE_DT
        assert "min_dt = -" in mgcfd._lib.load().mgcfd_last_error().decode()
        with pytest.raises(mgcfd._lib.MgcfdError):
            s.run(1)
        got.append([s.fetch(l) for l in range(2)])
        s.close()
    for a, b in zip(*got):
        assert np.isfinite(a).all()
        if form == "mixed":
            np.testing.assert_array_equal(a, b)
        else:
            np.testing.assert_allclose(a, b, rtol=0, atol=2.0 ** -40 * np.abs(b).max())
    fine, coarse = got[0]
    up = levels[0].node_to_mg
    count = np.bincount(up, minlength=len(coarse))
    mean = np.stack([np.bincount(up, weights=fine[:, k], minlength=len(coarse)) for k in range(5)], 1) / count[:, None]
    np.testing.assert_allclose(coarse, mean, rtol=0, atol=2.0 ** -48 * np.abs(mean).max())


@pytest.mark.parametrize("form", ["mixed", "dw"])
def test_stop_rule_leaves_a_large_levels_state(form):
    """A served solve stops after its last V-cycle, whose prolongation has begun the
    next step: level 0 of 81^3 nodes is then in `old` alone.  The result is the
    state of a solver run for as many V-cycles, bit for bit."""
    levels = mgcfd.HostMesh.generate(81, 2, 4).levels()
    s = mgcfd.Solver(levels, 0.5, 3.0, precision=form)
    s.run(3)
    assert s.synchronize() == 0
    want = s.fetch(0)
    s.close()
    server = mgcfd.Server(max_active=2, precision=form, max_cycles=3)
    ident = server.submit(levels, 0.5, 3.0, want_result=True)
    server.drain()
    (record, got), = [(r, x) for r, x in server.poll() if r["id"] == ident]
    server.close()
    assert (record["status"], record["cycles"]) == (0, 3)
    np.testing.assert_array_equal(got, want)
