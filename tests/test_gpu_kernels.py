"""The stage and field kernels at the edges of their tiles and dispatch: the
tall and the low tile, the two elementwise passes and the general tile kernel
compute the same points, so they are compared with each other over sizes,
boundaries and options, and the diagnostics with numpy in 64 bits."""
import numpy as np
import pytest

import cases  # noqa: F401  (tests/golden on the path)
import make_folded
from conftest import ROOT, inner, relerr
from glemur_gb300 import BatchRelaxation, GlemurError, Relaxation, _abi, configs

pytestmark = pytest.mark.gpu

# partial and whole tiles of 32 x 12 and 32 x 4 columns, odd sizes (the last
# pair of a row is half a pair), three points in a direction, one plane a tile
SHAPES = [(3, 3, 3), (4, 5, 6), (33, 13, 9), (32, 12, 24), (31, 11, 7), (34, 25, 40), (65, 4, 5), (7, 66, 10)]
PERI = [(1, 1, 0), (0, 0, 0), (1, 0, 1), (0, 1, 0)]


def case(shape, peri, precision, pressure=False, inertia=False, method="Stokes", seed=0, amplitude=0.1):
    """A braid on a randomly moved grid (periodic ghosts as images)."""
    p = configs.random_braid(11 + seed, shape=shape, precision=precision)
    p.xPeri, p.yPeri, p.zPeri = peri
    if pressure:
        p.pressure, p.beta, p.p0Amp, p.p0Width = 1, p.rnd(0.1), p.rnd(0.5), p.rnd(2.0)
    p.inertia = int(inertia)
    p.set_str("jMethod", method)
    p = configs.derive(p)
    B0, xb = configs.init_state(p)
    sp = np.array([p.dx, p.dy, p.dz])
    rng = np.random.default_rng(seed)
    x = xb.astype(np.float64)
    x[1:-1, 1:-1, 1:-1] += rng.uniform(-amplitude, amplitude, size=x[1:-1, 1:-1, 1:-1].shape) * sp
    L = (p.Lx + p.dx, p.Ly + p.dy, p.Lz + p.dz)
    for axis, on in ((2, peri[0]), (1, peri[1]), (0, peri[2])):
        if on:
            lo = np.take(x, -2, axis).copy()
            lo[..., 2 - axis] -= L[2 - axis]
            hi = np.take(x, 1, axis).copy()
            hi[..., 2 - axis] += L[2 - axis]
            ix = [slice(None)] * 4
            ix[axis] = 0
            x[tuple(ix)] = lo
            ix[axis] = -1
            x[tuple(ix)] = hi
    return p, x.astype(p.real_dtype()), B0


def stages(p, x, B0, kernel):
    q = p.copy()
    q.stageKernel = kernel
    g = Relaxation(q)
    g.upload(x, B0, 0.0, 1e-3)
    if p.inertia:
        g.upload_u(0.01 * np.random.default_rng(5).normal(size=g.I + (3,)))
    out = {}
    for n in range(6):
        g.stage(n)
        if n < 5:
            out[f"k{n}"] = g.k(n)
            out[f"x{n}"] = g.x(n)
    out["xnew"] = g.x(6)
    if p.inertia:
        out["unew"] = g.u(6)
    g.control()
    s = g.state()
    g.close()
    return out, s


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("peri", PERI)
@pytest.mark.parametrize("shape", SHAPES)
def test_stage_matches_the_general_kernel(shape, peri, precision):
    """Every stage's increments and grids, ghosts included: FP64 to rounding,
    FP32 within the 1e-5 per stage of the parity tests."""
    a, sa = stages(*case(shape, peri, precision), 0)
    b, sb = stages(*case(shape, peri, precision), 1)
    tol = 1e-12 if precision == 64 else 1e-5
    for name in a:
        assert relerr(a[name], b[name]) < tol, name
    assert sa["status"] == sb["status"] and sa["timeIndex"] == sb["timeIndex"]


@pytest.mark.parametrize("precision,form", [(p, f) for p in (32, 64) for f in
                                            ("pressure", "inertia", "inertia_pressure", "Stokes4th", "StokesQuint",
                                             "Classic", "Classic_pressure", "Classic_inertia")])
@pytest.mark.parametrize("shape,peri", [((33, 13, 9), (1, 1, 0)), ((20, 24, 17), (0, 0, 0)), ((3, 40, 12), (0, 1, 1))])
def test_options_match_the_general_kernel(shape, peri, precision, form):
    """As above with the pressure gradient and the Classic current (second differences
    of the positions: 1e-3 in FP32, as in the large case's parity test), the velocity
    equation and the currents with a kernel of their own."""
    method = "Classic" if form.startswith("Classic") else form if form.startswith("Stokes") else "Stokes"
    kw = dict(pressure="pressure" in form, inertia="inertia" in form, method=method)
    a, _ = stages(*case(shape, peri, precision, **kw), 0)
    b, _ = stages(*case(shape, peri, precision, **kw), 1)
    second = kw["pressure"] or method == "Classic"
    tol = 1e-12 if precision == 64 else (1e-3 if second else 1e-5)
    if precision == 64 and second:
        tol = 1e-10            # the same noise at FP64 rounding
    for name in a:
        assert relerr(a[name], b[name]) < tol, name


@pytest.mark.parametrize("precision", [32, 64])
def test_batched_and_single_runs_agree_bit_for_bit_on_odd_sizes(precision):
    """The batch's tall tile against the single case's low tile (FP32) and
    elementwise passes (FP64)."""
    cs = [case(s, p, precision, seed=i) for i, (s, p) in enumerate([((33, 13, 9), (1, 1, 0)), ((34, 25, 40), (0, 0, 0)),
                                                                   ((5, 66, 10), (0, 1, 1)), ((64, 24, 12), (1, 1, 0))])]
    b = BatchRelaxation([p for p, _, _ in cs])
    for i, (p, x, B0) in enumerate(cs):
        b.upload(i, x, B0, 0.0, 1e-3)
    b.steps_async(4)
    for i, (p, x, B0) in enumerate(cs):
        g = Relaxation(p)
        g.upload(x, B0, 0.0, 1e-3)
        g.steps_async(4)
        assert g.state() == b.state(i)
        assert np.array_equal(g.grid(), b.download(i)["xb"])
        g.close()
    b.close()


def test_sheared_cells_keep_their_precision_in_fp32():
    """Random displacements of 0.45 spacings: many determinants cancel and are
    recomputed in double.  Against the FP64 increments of the same grid the
    pair kernel is no further off than the general one (up to rounding)."""
    p, x, B0 = case((40, 30, 21), (1, 1, 0), 32, amplitude=0.45)
    q = p.copy()
    q.precision, q.errMode = 64, 1
    ref, _ = stages(q, x.astype(np.float64), B0.astype(np.float64), 1)
    new, _ = stages(p, x, B0, 0)
    old, _ = stages(p, x, B0, 1)
    err = lambda a: float(np.median(np.abs(a["k0"] - ref["k0"]) / (np.abs(ref["k0"]) + 1e-12)))  # noqa: E731
    assert err(new) <= 1.5 * err(old) + 1e-7
    norm = lambda a: float(np.linalg.norm((a["k0"] - ref["k0"]).ravel()) / np.linalg.norm(ref["k0"].ravel()))  # noqa: E731
    assert norm(new) <= 1.5 * norm(old) + 1e-6


@pytest.mark.parametrize("method", make_folded.METHODS)
def test_currents_on_the_folded_grid_match_the_fixture(method):
    """J of every current on the folded grid against the values stored from the
    reference's kernels (corner triangles, NaN points included)."""
    z = np.load(ROOT / "tests" / "golden" / "folded_currents.npz")
    p, _, _ = make_folded.folded_case(method)
    g = Relaxation(p)
    g.upload(z["x"], z["B0"])
    g.refresh()
    f = g.download()
    Jr = z[f"J_{method}"]
    assert np.array_equal(np.isnan(f["J"]), np.isnan(Jr))
    assert relerr(np.nan_to_num(f["J"]), np.nan_to_num(Jr)) < 1e-10
    assert relerr(inner(f["B"]), z["B"]) < 1e-12
    g.close()


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("shape,peri,scale", [((33, 20, 17), (1, 1, 0), 1.0), ((12, 12, 12), (0, 0, 0), 1.0),
                                              ((24, 16, 20), (1, 1, 1), 1e-13), ((24, 16, 20), (1, 1, 0), 0.0)])
def test_reductions_match_numpy_in_64_bits(shape, peri, scale, precision):
    """The sums and maxima of gm_refresh against numpy on the downloaded B, J and
    Delta; with scaled blobs J is far below the range of the FP32 pairs, or
    zero.  Sums of up to 11,000 non-negative terms: 1e-12."""
    p, x, B0 = case(shape, peri, precision)
    B0[..., :2] *= scale
    if scale < 1:                     # no grid noise: J comes from B0 alone
        _, x = configs.init_state(p)
    g = Relaxation(p)
    g.upload(x, B0)
    r = g.refresh()
    f = g.download()
    B, J, D = inner(f["B"]).astype(np.float64), f["J"].astype(np.float64), f["detJac"].astype(np.float64)
    jn, bn = np.linalg.norm(J, axis=-1), np.linalg.norm(B, axis=-1)
    cn = np.linalg.norm(np.cross(J, B), axis=-1)
    w = np.ones(D[1:-1, 1:-1, 1:-1].shape)
    for a in range(3):
        for e in (0, -1):
            ix = [slice(None)] * 3
            ix[a] = e
            w[tuple(ix)] *= 0.5
    both = jn * bn
    pw = np.divide(cn, both, out=np.zeros_like(cn), where=both > 0)
    b2 = (inner(f["B"]) ** 2).sum(-1, dtype=p.real_dtype()).astype(np.float64)
    want = dict(BMax=bn.max(), JMax=jn.max(), residual=cn.sum() / both.sum() if both.sum() > 0 else 0.0, residualPw=pw.mean(),
                errB_1ez=np.sqrt(((B - [0, 0, 1]) ** 2).sum(-1).mean()))
    for k, v in want.items():
        assert abs(r[k] - v) <= 1e-12 * max(abs(v), 1e-300) + 1e-30, (k, r[k], v)
    assert abs(r["B2"] / ((b2 * inner(D) * w).sum() * p.dx * p.dy * p.dz) - 1) < (1e-12 if precision == 64 else 1e-6)
    faces = [D[1:-1, 1:-1, 1:-1]]
    for a, on in ((2, peri[0]), (1, peri[1]), (0, peri[2])):
        if not on:
            ix = [slice(1, -1)] * 3
            for e in (0, -1):
                ix[a] = e
                faces.append(D[tuple(ix)])
    assert r["minDetJac"] == min(v.min() for v in faces)
    g.close()


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("shape", SHAPES)
def test_uploaded_grids_are_the_callers(shape, precision):
    """All four grids of a handle hold the uploaded points, ghosts included."""
    p, x, B0 = case(shape, (1, 1, 0), precision)
    g = Relaxation(p)
    g.upload(x, B0, 0.0, 1e-3)
    for which in (0, 1, 5, 6):
        np.testing.assert_array_equal(g.x(which), x)
    g.close()


@pytest.mark.parametrize("precision", [32, 64])
def test_set_time_in_stream_order(precision):
    """Between steps in flight: the state is changed where the call stands, what it
    does not name is kept, and a step size at the lower bound stops the steps."""
    p, x, B0 = case((20, 18, 22), (1, 1, 0), precision)
    g, h = Relaxation(p), Relaxation(p)
    for q in (g, h):
        q.upload(x, B0, 0.0, 1e-3)
    for _ in range(3):
        g.steps_async(1)
        g.set_time(0.5, 2e-3, 7)
    for _ in range(3):
        h.steps_async(1)
        n = h.state()["nAttempted"]
        h.set_time(0.5, 2e-3, 7)
        assert h.state()["nAttempted"] == n
    np.testing.assert_array_equal(g.grid(), h.grid())
    s, dt = g.state(), p.rnd(2e-3) if p.errMode == 0 else 2e-3      # errMode 0 keeps t and dt in REAL
    assert (s["t"], s["dt"], s["timeIndex"]) == (0.5, dt, 7) and s["nAttempted"] == 3
    g.set_time(0.5, p.dtMin)
    g.steps_async(2)
    assert g.state()["nAttempted"] == 3
    for q in (g, h):
        q.close()


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("peri", PERI + [(1, 1, 1)])
@pytest.mark.parametrize("shape", [(3, 4, 5), (33, 13, 9)])
def test_exported_ghosts_are_the_wrapped_points(shape, peri, precision):
    """Faces, edges and corners: one face pair after the other in the order z, y, x."""
    p, x, B0 = case(shape, peri, precision)
    g = Relaxation(p)
    g.upload(x, B0, 0.0, 1e-3)
    g.refresh()
    d = g.download()
    g.close()
    for f in (d["B"], d["detJac"]):
        w = f.copy()
        for axis, on in ((0, peri[2]), (1, peri[1]), (2, peri[0])):
            if on:
                v = np.moveaxis(w, axis, 0)
                v[0], v[-1] = v[-2].copy(), v[1].copy()
        np.testing.assert_array_equal(f, w)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("scale", [2.0 ** -33, 2.0 ** -30, 2.0 ** -24, 2.0 ** -20])
def test_reductions_of_a_weak_current_keep_their_bits(scale, precision):
    """J of 1e-10 to 1e-6 along a field that it turns by as little, so |J x B| is of the order
    of J^2 and its square near the lower end of single precision.  A grid of exact
    spacings, so J comes from B0 alone.  The terms are off by a few roundings of a double
    and the sums by as many as the reduction tree is deep (12): 20 of 2^-53, and the
    maxima, a root of a sum of three squares, by 1 ulp."""
    p = configs.random_braid(1, shape=(17, 9, 25), precision=precision)
    p.xPeri = p.yPeri = 0
    p = configs.derive(p)
    B0, x = configs.init_state(p)
    B0[..., 0], B0[..., 1], B0[..., 2] = -scale * x[..., 1], scale * x[..., 0], 1
    g = Relaxation(p)
    g.upload(x, B0)
    r = g.refresh()
    f = g.download()
    g.close()
    B, J = (a.astype(np.longdouble) for a in (inner(f["B"]), f["J"]))
    jn, bn = np.sqrt((J * J).sum(-1)), np.sqrt((B * B).sum(-1))
    cn = np.sqrt((np.cross(J, B) ** 2).sum(-1))
    assert 1e-10 < float(jn.max()) < 1e-5 and float(cn.max()) < 10 * float(jn.max()) ** 2
    want = dict(residual=cn.sum() / (jn * bn).sum(), residualPw=(cn / (jn * bn)).mean())
    for k, v in want.items():
        assert abs(r[k] / v - 1) < 20 * 2.0 ** -53, (k, r[k], v)
    for k, v in dict(BMax=bn.max(), JMax=jn.max()).items():
        assert abs(r[k] / v - 1) <= 2.0 ** -52, (k, r[k], v)


@pytest.mark.parametrize("shape", [(33, 20, 17), (24, 26, 40)])
def test_exported_b_and_delta_are_as_exact_as_the_plain_formula(shape):
    """FP64: the error of the exported B and Delta against extended precision, in the norm,
    is that of the same formula (Jacobian, its determinant, one reciprocal) evaluated in
    doubles, up to the sampling of some 30,000 roundings and their FMAs: 15 %."""
    p, x, B0 = case(shape, (1, 1, 0), 64)
    g = Relaxation(p)
    g.upload(x, B0)
    g.refresh()
    f = g.download()
    g.close()

    def plain(real):
        q, b = x.astype(real), inner(B0).astype(real)
        ends = [(q[1:-1, 1:-1, 2:], q[1:-1, 1:-1, :-2]), (q[1:-1, 2:, 1:-1], q[1:-1, :-2, 1:-1]), (q[2:, 1:-1, 1:-1], q[:-2, 1:-1, 1:-1])]
        j = [(hi - lo) * (real(1) / real(d) / 2) for (hi, lo), d in zip(ends, (p.dx, p.dy, p.dz))]       # j[a][..., l]
        m = lambda l, a: j[a][..., l]  # noqa: E731
        D = (m(0, 0) * m(1, 1) * m(2, 2) + m(0, 1) * m(1, 2) * m(2, 0) + m(0, 2) * m(1, 0) * m(2, 1)
             - m(0, 0) * m(1, 2) * m(2, 1) - m(0, 1) * m(1, 0) * m(2, 2) - m(0, 2) * m(1, 1) * m(2, 0))
        return np.stack([sum(m(l, a) * b[..., a] for a in range(3)) * (1 / D) for l in range(3)], -1), D

    (B, D), (Bx, Dx) = plain(np.float64), plain(np.longdouble)
    off = lambda a, e: float(np.linalg.norm((a - e).astype(np.float64).ravel()) / np.linalg.norm(e.astype(np.float64).ravel()))  # noqa: E731
    assert off(inner(f["B"]), Bx) < 1.15 * off(B, Bx)
    assert off(inner(f["detJac"]), Dx) < 1.15 * off(D, Dx)


def test_runs_without_tiles_have_nothing_to_tune():
    """FP64 runs by the field passes: the autotuner launches nothing and returns the depth
    chosen at creation, which can be set again (and any other within 1..nz) without
    changing the run; a tile run is timed, and a run the tile kernel cannot do
    refuses a depth."""
    p, x, B0 = case((20, 18, 22), (1, 1, 0), 64)
    grids = []
    for tune in (False, True):
        g = Relaxation(p)
        g.upload(x, B0, 0.0, 1e-3)
        if tune:
            n = g.launches
            r = g.autotune(2)
            assert g.launches == n and r["ms_stages_0_4"] == 0 and 1 <= r["tz"] <= p.nz
            g.steps_async(1)
            for tz in (r["tz"], 1, p.nz):
                g.set_tile_z(tz)
            for tz in (0, p.nz + 1):
                with pytest.raises(GlemurError):
                    g.set_tile_z(tz)
            g.steps_async(2)
        else:
            g.steps_async(3)
        grids.append(g.grid())
        g.close()
    np.testing.assert_array_equal(*grids)
    p, x, B0 = case((20, 18, 22), (1, 1, 0), 32)
    g = Relaxation(p)
    g.upload(x, B0, 0.0, 1e-3)
    n = g.launches
    assert g.autotune(2)["ms_stages_0_4"] > 0 and g.launches > n
    g.close()
    p, x, B0 = case((20, 18, 22), (1, 1, 0), 32, inertia=True)
    g = Relaxation(p)
    g.upload(x, B0, 0.0, 1e-3)
    with pytest.raises(GlemurError):
        g.set_tile_z(4)
    g.close()


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("what", ["no_current", "aligned", "tiny_field", "not_a_number", "infinite"])
def test_reductions_of_zeros_and_what_is_not_finite(what, precision):
    """On a grid of exact spacings: a current of zero, one along the field, a field whose
    squares underflow in FP32, and a point that is not finite: sums as numpy's on the
    downloaded fields (NaN where theirs is), maxima that leave NaN out."""
    p = configs.random_braid(1, shape=(17, 9, 25), precision=precision)
    p.xPeri = p.yPeri = 0
    p = configs.derive(p)
    B0, x = configs.init_state(p)
    B0[...] = (0, 0, 1)
    if what == "aligned":
        B0[..., 0], B0[..., 1] = -0.25 * x[..., 1], 0.25 * x[..., 0]
        B0[..., 2] = 0
    if what == "tiny_field":
        B0 *= 2.0 ** -70
        B0[..., 0] = 2.0 ** -72 * np.sin(x[..., 1])
    if what in ("not_a_number", "infinite"):
        B0[12, 5, 8, 1] = np.nan if what == "not_a_number" else np.inf
    g = Relaxation(p)
    g.upload(x, B0)
    r = g.refresh()
    f = g.download()
    g.close()
    B, J = (a.astype(np.float64) for a in (inner(f["B"]), f["J"]))
    with np.errstate(all="ignore"):
        jn, bn = np.sqrt((J * J).sum(-1)), np.sqrt((B * B).sum(-1))
        cn = np.sqrt((np.cross(J, B) ** 2).sum(-1))
        both = jn * bn
        pw = np.where(both > 0, cn / both, 0)
        want = dict(residual=cn.sum() / both.sum() if both.sum() > 0 or np.isnan(both.sum()) else 0.0, residualPw=pw.mean(),
                    BMax=np.nanmax(bn), JMax=np.nanmax(jn))
    if what == "no_current":
        assert want["JMax"] == 0
    for k, v in want.items():
        if np.isfinite(v):
            assert abs(r[k] - v) <= 1e-13 * abs(v), (k, r[k], v)
        elif k in ("BMax", "JMax"):
            assert r[k] == v, (k, r[k], v)
        else:
            assert not np.isfinite(r[k]) or (k == "residual" and r[k] == 0), (k, r[k], v)


@pytest.mark.parametrize("name", ["braid_f64", "tied_f64", "zperi_f64", "shear_f64", "centershift_tied_f64", "oct_tied_f64", "braid_f32",
                                  "shear_f32"])
def test_refresh_matches_the_oracle_on_every_face(name):
    """What gm_refresh exports, the ghost faces with it: periodic, line-tied, and line-tied on
    an initially distorted grid."""
    from oracle.pyoracle import Oracle
    p = cases.make(name)
    B0, x = configs.init_state(p)
    d = np.array([p.dx, p.dy, p.dz])
    x[1:-1, 1:-1, 1:-1] += (0.2 * np.random.default_rng(3).uniform(-1, 1, size=inner(x).shape) * d).astype(x.dtype)
    for axis, peri, L in ((2, p.xPeri, p.Lx + p.dx), (1, p.yPeri, p.Ly + p.dy), (0, p.zPeri, p.Lz + p.dz)):
        if peri:                         # the ghosts of a periodic face are the images
            v = np.moveaxis(x, axis, 0)
            v[0], v[-1] = v[-2], v[1]
            v[0, ..., 2 - axis] -= x.dtype.type(L)
            v[-1, ..., 2 - axis] += x.dtype.type(L)
    g, o = Relaxation(p), Oracle(p, B0, x)
    g.upload(x, B0)
    g.refresh()
    o.refresh()
    f, w = g.download(), o.get()
    g.close()
    o.close()
    tol = 1e-12 if p.precision == 64 else 1e-5
    assert relerr(inner(f["B"]), inner(w["B"])) < tol and relerr(f["J"], w["J"]) < 50 * tol
    assert relerr(inner(f["detJac"]), inner(w["detJac"])) < tol
    for axis, peri in ((0, p.zPeri), (1, p.yPeri), (2, p.xPeri)):
        for side in (0, -1):
            ix = [slice(1, -1)] * 3
            ix[axis] = side
            for k in ("B", "detJac"):
                assert relerr(f[k][tuple(ix)], w[k][tuple(ix)]) < tol, (axis, side, k)
