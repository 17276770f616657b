"""Kernel variants chosen by a rule on sizes, at the sizes where the rule or
the variant can go wrong (GPU)."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

import mgcfd
from irregular import irregular_levels
from mgcfd import _build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed", "dw"])
@pytest.mark.parametrize("axes", [(3, 3, 3, 3, 3, 3, 4), (8, 8), (5, 8, 3, 16, 4), (9,)])
def test_batch_norms_blocks_within_and_across_meshes(precision, axes):
    """The level-0 norms of a batch, where a block of 128 nodes lies in one
    mesh (8^3 = 4 whole blocks), spans several (27 nodes each) or ends a level,
    against each mesh solved alone.  The states agree to rounding (a few
    1e-16), the residuals are their differences, 1e-7 and more of the state:
    a node's residual agrees to 1e-8 relative, and so do the norms.  A norm that
    missed or double-counted one of at most 4096 nodes is off by 1e-4 or so."""
    meshes = [mgcfd.HostMesh.generate(n, 1, 40 + k) for k, n in enumerate(axes)]
    machs = [0.3 + 0.05 * k for k in range(len(axes))]
    batch = mgcfd.Batch(meshes, machs, [2.0] * len(axes), precision=precision)
    batch.run(3)
    assert batch.synchronize() == 0
    for k, m in enumerate(meshes):
        solo = mgcfd.Solver(m, machs[k], 2.0, precision=precision)
        solo.run(3)
        st, rms, rho = solo.norms()
        bst, brms, brho = batch.mesh_status(k)
        assert (st, bst) == (0, 0)
        np.testing.assert_allclose([brms, brho], [rms, rho], rtol=1e-6, atol=0)
        solo.close()
    batch.close()


def _ulps(x, exact):
    """|x - exact| in units of the last place of exact (exact: long double)."""
    _, e = np.frexp(exact.astype(np.float64))
    return np.abs(x.astype(np.longdouble) - exact) * np.ldexp(np.longdouble(1), 53 - e)


def _seed_inputs(kind):
    rng = np.random.default_rng(11)
    n = 400_000
    if kind == "mantissas":  # every exponent of the fast range and beyond its ends
        b = np.ldexp(1.0 + rng.random(n), rng.integers(-64, 64, n))
    elif kind == "near_powers":  # a few units around every power of two, and around FP32 rounding ties
        k = rng.integers(-61, 62, n)
        b = np.ldexp(1.0, k) * (1.0 + rng.integers(-40, 41, n) * 2.0 ** -53)
        tie = rng.random(n) < 0.5
        f = rng.integers(0, 1 << 23, n) * 2.0 ** -23 + 2.0 ** -24
        b = np.where(tie, np.ldexp(1.0 + f, k) * (1.0 + rng.integers(-3, 4, n) * 2.0 ** -52), b)
    else:  # results next to a power of two, from both sides
        k = rng.integers(-59, 60, n)
        r = np.ldexp(1.0, k // 2) * (1.0 + rng.integers(-2000, 2001, n) * 2.0 ** -rng.integers(22, 53, n))
        b = np.where(rng.random(n) < 0.5, 1.0 / r, r * r)
    a = np.ldexp(1.0 + rng.random(n), rng.integers(-300, 300, n)) * rng.choice([-1.0, 1.0], n)
    return a, b


@pytest.fixture(scope="module")
def native():
    here = Path(__file__).resolve().parent
    out = here / "_build" / "libseed_check.so"
    out.parent.mkdir(exist_ok=True)
    subprocess.run([_build._nvcc(), *_build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    f"-I{_build.CSRC}", str(here / "native" / "seed_check.cu"), "-o", str(out)], check=True,
                   capture_output=True)
    return C.CDLL(str(out))


@pytest.fixture(scope="module")
def seed_check(native):
    def run(a, b):
        outs = [np.empty(len(b)) for _ in range(4)]
        p = [x.ctypes.data_as(C.c_void_p) for x in (a, b, *outs)]
        assert native.seed_check(C.c_int64(len(b)), *p) == 0
        return outs

    return run


@pytest.mark.parametrize("kind", ["mantissas", "near_powers", "near_power_results"])
def test_seeded_reciprocal_quotient_root(seed_check, kind):
    """rcp_fast, div_fast and sqrt_fast against long double.  The seeds are
    within 2^-42, so one Newton step leaves 0.5 ulp of rounding and, for the
    root, 2^-42 * 2^-21 * 2^53 = 2^-10 ulp more: 0.5 + 2^-9 is the bound."""
    a, b = _seed_inputs(kind)
    r, q, s, by = seed_check(a, b)
    A, B = a.astype(np.longdouble), b.astype(np.longdouble)
    slack = 0.5 + 2.0 ** -9
    assert _ulps(r, 1 / B).max() <= slack
    assert _ulps(q, A / B).max() <= slack
    assert _ulps(s, np.sqrt(B)).max() <= slack
    fast = (b >= 2.0 ** -60) & (b < 2.0 ** 60)
    np.testing.assert_array_equal(by[fast], (a / b)[fast])  # the set-up's quotients are the host's, bit for bit


def test_seeded_forms_keep_the_ieee_special_cases(seed_check):
    """Operands outside the fast range give the IEEE result bit for bit; the
    ones just inside it (2^-60 and the number below 2^60, whose reciprocal and
    root lie 2^-53 ulp from a rounding tie) are held to the bound above."""
    edge = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.2e-308, 1.7e308, -1.0, -4.0, 2.0 ** -60,
                     2.0 ** 60, np.nextafter(2.0 ** 60, 0), np.nextafter(2.0 ** -60, 0), 2.0 ** -61, 1e-200, 1e200])
    a, b = (x.ravel().copy() for x in np.meshgrid(edge, edge))
    r, q, s, by = seed_check(a, b)
    fast_b = (b >= 2.0 ** -60) & (b < 2.0 ** 60)
    fast_q = fast_b & (np.abs(a) >= 2.0 ** -900) & (np.abs(a) < 2.0 ** 900)
    with np.errstate(all="ignore"):
        want = [1.0 / b, a / b, np.sqrt(b)]
        exact = [1 / b.astype(np.longdouble), a.astype(np.longdouble) / b, np.sqrt(b.astype(np.longdouble))]
    for got, w, ld, fast in zip((r, q, s), want, exact, (fast_b, fast_q, fast_b)):
        nan = np.isnan(w)
        assert np.isnan(got[nan]).all()
        ieee = ~nan & ~fast
        assert np.array_equal(got[ieee].view(np.uint64), w[ieee].view(np.uint64))
        assert _ulps(got[fast], ld[fast]).max() <= 0.5 + 2.0 ** -9
    # (div_by may miss a quotient within 2^-52 ulp of a tie: powers of two by the number below 2^60 are)
    finite = np.isfinite(a) & ~np.isnan(want[1]) & (b != np.nextafter(2.0 ** 60, 0))
    assert np.array_equal(by[finite].view(np.uint64), want[1][finite].view(np.uint64))


@pytest.mark.parametrize("terms", [1, 2, 6, 7, 14, 40])
def test_sum32_is_no_worse_than_fp64_adds(native, terms):
    """Sum32 over FP32 terms of both signs and of magnitudes 2^40 apart,
    cancelling ones among them: within half an ulp of the exact sum plus
    n^2 2^-72 of the terms' magnitudes (and the two roundings of lo + tail and
    of the value: 2^-53 of a result, 2^-24 * 2^-53 of the magnitudes), which is no
    more than adding the widened terms one by one in FP64 may lose."""
    rng = np.random.default_rng(terms)
    n = 100_000
    x = np.ldexp(rng.random((n, terms)) * 2 - 1, rng.integers(-20, 21, (n, terms))).astype(np.float32)
    k = terms // 2
    x[: n // 2, k:2 * k] = -x[: n // 2, :k] * np.float32(1 + 2.0 ** -20)
    out = np.empty(n)
    assert native.sum_check(C.c_int64(n), C.c_int(terms), x.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p)) == 0
    exact = x.astype(np.longdouble).sum(axis=1)
    mag = np.abs(x).astype(np.longdouble).sum(axis=1)
    err = np.abs(out.astype(np.longdouble) - exact)
    # (long double sums of the references: 64 significand bits or more, 2^-63 of the magnitudes)
    bound = np.abs(exact) * 2.0 ** -53 + mag * (terms ** 2 * 2.0 ** -72 + 2.0 ** -77 + terms * 2.0 ** -63)
    assert (err <= bound).all()
    seq = np.zeros(n)
    for j in range(terms):
        seq = seq + x[:, j].astype(np.float64)
    assert err.sum() <= np.abs(seq.astype(np.longdouble) - exact).sum() * (1 + 1e-9) + float(bound.sum()) * 1e-3


@pytest.mark.parametrize("terms", [41, 300, 1700])
@pytest.mark.parametrize("signs", ["one", "both"])
def test_sum32_of_many_terms(native, terms, signs):
    """... and for nodes with many edges: n^3/6 2^-72 of the terms' magnitudes (each
    of the three words' rounding added up), half an ulp of the value, and 2^-53 of
    lo + tail, itself n 2^-24 of the magnitudes."""
    rng = np.random.default_rng(terms)
    n = 4_000
    x = rng.random((n, terms)) if signs == "one" else rng.random((n, terms)) * 2 - 1
    x = x.astype(np.float32)
    out = np.empty(n)
    assert native.sum_check(C.c_int64(n), C.c_int(terms), x.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p)) == 0
    exact = x.astype(np.longdouble).sum(axis=1)
    mag = np.abs(x).astype(np.longdouble).sum(axis=1)
    bound = np.abs(exact) * 2.0 ** -53 + mag * (terms ** 3 / 6 * 2.0 ** -72 + terms * 2.0 ** -77 + terms * 2.0 ** -63)
    assert (np.abs(out.astype(np.longdouble) - exact) <= bound).all()


def test_sum32_beyond_binary32_and_not_finite(native):
    f = np.float32
    x = np.array([[np.inf, 1], [-np.inf, 1], [np.inf, -np.inf], [np.nan, 1], [3e38, 3e38], [-3e38, -3e38], [0.0, -0.0],
                  [1e-40, 2e-40]], dtype=f)
    out = np.empty(len(x))
    assert native.sum_check(C.c_int64(len(x)), C.c_int(2), x.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p)) == 0
    np.testing.assert_array_equal(out[:2], [np.inf, -np.inf])
    assert np.isnan(out[2:4]).all()
    np.testing.assert_array_equal(out[4:6], [np.inf, -np.inf])  # leaves binary32's range
    assert out[6] == 0.0
    assert out[7] == float(x[7, 0]) + float(x[7, 1])


def _small_levels(kind):
    if kind == "irregular":  # up to fifteen or so edges at a node: two rounds of eight
        return irregular_levels(1500, 3, 3)
    if kind == "hub":  # one node with forty edges: five rounds and a ragged one
        levels = irregular_levels(300, 1, 8)
        L = levels[0]
        e = np.stack([np.full(40, 7), np.arange(40, 80)], 1).astype(np.int32)
        d = L.coords[e[:, 1]] - L.coords[e[:, 0]]
        L.edge_to_nodes = np.ascontiguousarray(np.concatenate([L.edge_to_nodes, e]))
        L.edge_weights = np.ascontiguousarray(np.concatenate([L.edge_weights, 0.02 * d]))
        return levels
    n = int(kind)
    return mgcfd.HostMesh.generate(n, min(3, max(1, n.bit_length() - 1)), 70 + n).levels()


# lattices: 8 nodes; ragged last blocks; the last level with eight threads per node and the
# first without for FP64 (16, 17), DW (20, 21) and mixed (25, 26)
@pytest.mark.parametrize("kind", ["2", "3", "5", "16", "17", "20", "21", "25", "26", "irregular", "hub"])
@pytest.mark.parametrize("form", ["fp64", "mixed", "pair32", "dw"])
def test_small_levels_equal_the_other_stage(kind, form):
    """Small levels (eight threads per node) against the same solve with
    k_update's stages: mixed precision against the gather increment and DW
    against a batch of the mesh and a copy, bit for bit; FP64 against the atomic
    increment, whose sums differ in order alone (a few 1e-16 of the state)."""
    levels = _small_levels(kind)
    opts = dict(precision="mixed", accumulation=form if form == "pair32" else "fp64") if form in ("mixed", "pair32") \
        else dict(precision=form)

    def solve(**more):
        s = mgcfd.Solver(levels, 0.55, 2.5, **opts, **more)
        s.run(2)
        assert s.synchronize() == 0
        out = [s.fetch(l) for l in range(len(levels))], s.norms()[1:]
        s.close()
        return out

    got, norms = solve()
    if form == "dw":
        b = mgcfd.Batch([levels, levels], [0.55, 0.55], [2.5, 2.5], **opts)
        b.run(2)
        assert b.synchronize() == 0
        want, wnorms = [b.fetch_mesh(1, l) for l in range(len(levels))], b.mesh_status(1)[1:]
        b.close()
    else:
        want, wnorms = solve(increment="atomic" if form == "fp64" else "gather")
    for l in range(len(levels)):
        if form == "fp64":
            np.testing.assert_allclose(got[l], want[l], rtol=0, atol=1e-13 * np.abs(want[l]).max())
        else:
            np.testing.assert_array_equal(got[l], want[l])
    np.testing.assert_allclose(norms, wnorms, rtol=1e-6, atol=0)


@pytest.mark.parametrize("n", [8, 30, 81])  # small levels throughout or below; a level 0 that keeps its begun state in one array
@pytest.mark.parametrize("form", ["mixed", "dw"])
def test_states_between_steps(n, form):
    """Every level's variables after every smoothing step and its transfer (the
    fused stage leaves a begun level's state in one array and a finished one's in
    another), against the gather increment: bit for bit in mixed precision; DW's
    gather sums in another form, within the pairs' 2^-42 of each variable's scale."""
    mesh = mgcfd.HostMesh.generate(n, 3, 5)
    a = mgcfd.Solver(mesh, 0.6, 2.0, precision=form)
    b = mgcfd.Solver(mesh, 0.6, 2.0, precision=form, increment="gather")
    for _ in range(9):  # two V-cycles of four steps and one step more
        assert a.step() == b.step()
        for l in range(3):
            x, y = a.fetch(l), b.fetch(l)
            if form == "mixed":
                np.testing.assert_array_equal(x, y)
            else:
                np.testing.assert_allclose(x, y, rtol=0, atol=2.0 ** -42 * np.abs(y).max())
    a.close()
    b.close()


@pytest.mark.parametrize("form", ["mixed", "dw"])
def test_small_restriction_equals_the_other(form):
    """Restriction with eight threads per coarse node (plain solvers) against a
    batch's, bit for bit: random maps with up to a dozen and more children per
    coarse node (two rounds), coarse nodes without any, and the level-0 norms."""
    levels = irregular_levels(4000, 3, 21)
    solo = mgcfd.Solver(levels, 0.5, 1.0, precision=form)
    pair = mgcfd.Batch([levels, levels], [0.5, 0.5], [1.0, 1.0], precision=form)
    for s in (solo, pair):
        s.run(2)
        assert s.synchronize() == 0
    for l in range(3):
        np.testing.assert_array_equal(solo.fetch(l), pair.fetch_mesh(0, l))
    np.testing.assert_allclose(solo.norms()[1:], pair.mesh_status(0)[1:], rtol=1e-6, atol=0)
    solo.close()
    pair.close()
