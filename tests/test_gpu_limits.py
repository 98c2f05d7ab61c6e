"""Where the float pairs and triples of the FP64 paths end: results that leave
the floats' range, values that are not numbers, thresholds and faces met to
the last bits, rays and requests handed to binary64.  Against the oracle at
the bars of the other tests (FP64 images 1e-8 a conditioned pixel, fluid
scalars 1e-12, synchrotron 1e-11).
"""

import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu

KW = dict(mass_scale=3e26, M_bh=6.5e9 * 1.989e33, r_high=40, max_nsteps=3000)


def _np(t):
    return t.detach().cpu().numpy()


def _model(arrs):
    from mahakala_gb300.grmhd.athenak import AthenakFluidModel
    return AthenakFluidModel(arrs, arrs.bhspin, fluid_gamma=13. / 9)


# rescale_nu = 1 (the default) leaves the emissivity divided by nu^2: down to
# 1e-50 in the units the triples use
@pytest.mark.parametrize("rescale_nu", [1.0, 7.0, 1 / 230e9, 1e-17])
def test_synchrotron_invariants_of_any_scale(cuda, orc, rescale_nu):
    import mahakala_gb300 as mk
    rng = np.random.default_rng(4)
    n = 20000
    args = [10.0 ** rng.uniform(-100, 12, n), 10.0 ** rng.uniform(np.log10(0.3), 6, n), 10.0 ** rng.uniform(-6, 8, n),
            np.arccos(rng.uniform(-1, 1, n)), 10.0 ** rng.uniform(3, 16, n)]
    with np.errstate(all="ignore"):
        refs = orc.synchrotron_coefficients(*args, rescale_nu=rescale_nu)
    for x, ref in zip(mk.synchrotron_coefficients(*args, rescale_nu=rescale_nu), refs):
        x = _np(x)
        assert np.array_equal(np.isnan(x), np.isnan(ref)) and np.array_equal(np.isinf(x), np.isinf(ref))
        ok = np.isfinite(ref) & (np.abs(ref) > 1e-290)
        assert ok.sum() > 2000 and np.max(rel_err(x[ok], ref[ok])) < 1e-11


def test_synchrotron_default_rescaling_golden(cuda):
    """The reference's own values at rescale_nu = 1, its default."""
    import mahakala_gb300 as mk
    from conftest import golden
    d = golden("synchrotron")
    em, ab = mk.synchrotron_coefficients(*(d[k] for k in ("Ne", "Theta", "B", "pitch", "nu")))
    assert np.max(rel_err(_np(em), d["em_inv1"])) < 1e-11 and np.max(rel_err(_np(ab), d["ab_inv1"])) < 1e-11


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("which", [(0,), (1,), (2,), (3,), (4,), (1, 3), (1, 2, 3), (5,), (5, 6, 7)])
def test_fluid_with_cells_that_are_not_finite(cuda, orc, which, value):
    """What such a cell reaches is not a number, as the reference has it."""
    from mahakala_gb300.grmhd.synthetic import make_synthetic_snapshot
    arrs = make_synthetic_snapshot(nblocks=2, cells_per_block=8, extent=20., bhspin=0.94)
    rng = np.random.default_rng(6)
    bad = rng.random(arrs.uov.shape[1:]) < 0.02
    for i in which:
        (arrs.uov[i] if i < 5 else arrs.B[i - 5])[bad] = value
    X = rng.uniform(-19, 19, (3000, 3))
    X = X[(X ** 2).sum(axis=1) > 4.0]
    S = np.concatenate([np.zeros((len(X), 1)), X, rng.normal(size=(len(X), 4))], 1)
    with np.errstate(all="ignore"):
        ref = orc.OracleSnapshot(arrs).get_fluid_scalars_from_geodesics(S)
    assert sum(np.isnan(v).sum() for v in ref.values()) > 100
    g = _model(arrs).get_fluid_scalars_from_geodesics(S)
    for k, x in g.items():
        x = _np(x)
        assert np.array_equal(np.isnan(x), np.isnan(ref[k])), k
        if k in ("dens", "u", "b"):
            assert np.array_equal(np.isinf(x), np.isinf(ref[k])), k
            ok = np.isfinite(ref[k])
            assert np.max(rel_err(x[ok], ref[k][ok])) < 1e-12, k


@pytest.mark.parametrize("extent", [20.0, 21.7, 30.1, 47.3])
def test_fluid_beside_cell_centres(cuda, orc, extent):
    """Points within float rounding of a cell's centre, either side; cells of
    like size, so that the oracle's 1e-15 of a weight is 1e-15 of the sum."""
    from mahakala_gb300.grmhd.synthetic import make_synthetic_snapshot
    arrs = make_synthetic_snapshot(nblocks=4, cells_per_block=8, extent=extent, bhspin=0.94)
    rng = np.random.default_rng(8)
    arrs.uov[:] = rng.uniform(1, 2, arrs.uov.shape)
    arrs.B[:] = rng.uniform(1, 2, arrs.B.shape)
    d = 2 * extent / 32
    X = (rng.integers(0, 32, (40000, 3)) + 0.5) * d - extent
    X += d * rng.uniform(-1.5e-7, 1.5e-7, X.shape)
    X = X[(X ** 2).sum(axis=1) > 4.0]
    S = np.concatenate([np.zeros((len(X), 1)), X, rng.normal(size=(len(X), 4))], 1)
    ref = orc.OracleSnapshot(arrs).get_fluid_scalars_from_geodesics(S)
    g = _model(arrs).get_fluid_scalars_from_geodesics(S)
    for k in ("dens", "u", "b"):
        assert np.nanmax(rel_err(_np(g[k]), ref[k])) < 1e-12, k


# thresholds whose first 24 bits, cut, leave more than half a unit behind, and
# some that do not: the distance decides to its last bits
@pytest.mark.parametrize("tol", [1e-3, 1e-4, 3e-3, 7.3e-4, 0.011])
def test_capture_radius_to_the_last_bits(cuda, orc, tol):
    from mahakala_gb300.geodesics import step_policy, trace
    eps = np.array([-1e-6, -1e-7, -3e-8, -1e-8, -1e-9, 1e-9, 1e-8, 3e-8, 1e-7, 1e-6])
    s0 = np.zeros((len(eps), 8))
    s0[:, 1] = 2.0 + tol * (1.0 + eps)
    s0[:, 4:6] = (1.0, -0.4)     # outward, traced back
    o = orc.integrate(s0, 4, 40.0, tol, 0.0)
    g = trace(s0, 0.0, step_policy(4, 40.0, tol))
    assert np.array_equal(o["K"] > 0, eps > 0)
    assert np.array_equal(_np(g["K"]), o["K"]) and np.array_equal(_np(g["why"]), o["why"])


@pytest.mark.parametrize("key", ["capture", "r_escape", "hmin", "hmax"])
def test_fixed_rule_to_the_last_bits(cuda, orc, key):
    """The fixed-fraction rule's thresholds at 1 +- 1e-8 of the value that
    decides: stops, and step sizes, on the right side."""
    from mahakala_gb300.geodesics import step_policy, trace
    rng = np.random.default_rng(12)
    for r0 in rng.uniform(20.0, 60.0, 24):
        s0 = np.zeros((1, 8))
        s0[:, 1] = r0
        s0[:, 4:6] = (1.0, 0.9) if key == "capture" else (1.0, -0.9)
        if key in ("capture", "r_escape"):
            r1 = orc.trace_fixed(s0, 1, 0.0)["state"][0, 1]
            value = r1 / 2.0 if key == "capture" else r1
        else:
            value = 0.05 * r0
        for e in (-1e-8, 1e-8):
            kw = {key: value * (1.0 + e)}
            if key == "hmin":
                kw["hmax"] = 100.0
            o = orc.trace_fixed(s0, 1, 0.0, **kw)
            g = trace(s0, 0.0, step_policy(1, kind="fixed", **kw))
            assert _np(g["why"])[0] == o["why"][0], (r0, e)
            assert np.max(rel_err(_np(g["state"]), o["state"], floor=1e-3)) < 1e-12, (r0, e)


def _without_block(arrs, m):
    import copy
    out, keep = copy.copy(arrs), np.arange(len(arrs.Levels)) != m
    out.uov, out.B = arrs.uov[:, keep], arrs.B[:, keep]
    for k in ("x1v", "x2v", "x3v", "x1f", "x2f", "x3f", "LogicalLocations", "Levels"):
        setattr(out, k, np.asarray(getattr(arrs, k))[keep])
    return out


def test_fluid_beside_a_missing_block(cuda, orc):
    """Points within float rounding of a block that the snapshot lacks."""
    from mahakala_gb300.grmhd.synthetic import make_synthetic_snapshot
    arrs = make_synthetic_snapshot(nblocks=4, cells_per_block=8, extent=20., bhspin=0.94)
    m = int(np.flatnonzero((np.asarray(arrs.LogicalLocations) == (0, 1, 2)).all(axis=1))[0])
    arrs = _without_block(arrs, m)      # x in (-20, -10], y in (-10, 0], z in (0, 10]
    rng = np.random.default_rng(9)
    X = rng.uniform((-20, -10, 0), (-10, 0, 10), (4000, 3))
    off = rng.choice([-1, 1], 4000) * 10.0 ** rng.uniform(-9, -6, 4000)
    side, axis = rng.integers(0, 2, 4000), rng.integers(0, 3, 4000)
    face = np.array([[-20, -10], [-10, 0], [0, 10]], float)
    X[np.arange(4000), axis] = face[axis, side] + off
    X = X[X[:, 0] > -20]
    S = np.concatenate([np.zeros((len(X), 1)), X, rng.normal(size=(len(X), 4))], 1)
    ref = orc.OracleSnapshot(arrs).get_fluid_scalars_from_geodesics(S)
    g = _model(arrs).get_fluid_scalars_from_geodesics(S)
    for k in ("dens", "u", "b"):
        assert np.nanmax(rel_err(_np(g[k]), ref[k])) < 1e-12, k


@pytest.mark.parametrize("extent", [20.0, 21.7, 30.1, 47.3])
def test_fp64_image_along_a_refinement_face(cuda, orc, extent):
    """A column of rays that run in the plane of a face between coarse and
    refined blocks: the point belongs to the block below (left < x <= right)."""
    from mahakala_gb300.grmhd.synthetic import make_multilevel_snapshot
    arrs = make_multilevel_snapshot(nblocks=2, cells_per_block=8, extent=extent, bhspin=0.0,
                                    refine=[(0, i, 1, k) for i in (0, 1) for k in (0, 1)])
    s0 = orc.initialize_geodesics_at_camera(0.0, 60.0, 1000, -10.0, 10.0, 5)
    # (the centre has no direction)
    assert (s0[10:15, 2] == 0).all() and (np.nan_to_num(s0[10:15, 6]) == 0).all()
    p = _image_parity(orc, arrs, 20.0, 5, 0.0)
    assert p["steps_equal"] and p["max_pixel_rel_err"] <= 1e-8, p


def _image_parity(orc, arrs, fov, res, spin, nu=230e9, **kw):
    from mahakala_gb300.images import RenderRequest, render_requests
    req = RenderRequest(_model(arrs), camera_inclination=60.0, fov=fov, resolution=res, bhspin=spin,
                        observing_frequency=nu, **dict(KW, **kw))
    img = _np(render_requests([req], with_steps=True)[0]).reshape(1, -1)
    s0 = orc.initialize_geodesics_at_camera(spin, 60.0, 1000, -fov / 2, fov / 2, res)
    osnap = orc.OracleSnapshot(arrs, bhspin=spin)
    with np.errstate(all="ignore"):
        ref, rsteps = orc.render_rays(osnap, s0, observing_frequency=nu, **dict(KW, **kw))
        pert, psteps = orc.render_rays(osnap, orc.perturbed(s0), observing_frequency=nu, **dict(KW, **kw))
    return orc.image_parity(img, _np(req.out["nsteps"]), ref, rsteps, pert, psteps)


@pytest.mark.parametrize("missing,off", [("y > 0", 1e-8), ("y < 0", -1e-8), ("y > 0", 3e-7)])
def test_fp64_image_beside_missing_blocks(cuda, orc, missing, off):
    """A column of rays in a plane beside the face where a snapshot ends."""
    from mahakala_gb300.grmhd.synthetic import make_synthetic_snapshot
    arrs = make_synthetic_snapshot(nblocks=4, cells_per_block=8, extent=20., bhspin=0.0)
    arrs.x2f, arrs.x2v = arrs.x2f + off, arrs.x2v + off
    # one far block of the missing side keeps the table's extent
    loc = np.asarray(arrs.LogicalLocations)
    gone = (loc[:, 1] >= 2) if missing == "y > 0" else (loc[:, 1] < 2)
    gone &= ~(loc == ((3, 3, 0) if missing == "y > 0" else (3, 0, 0))).all(axis=1)
    for m in np.flatnonzero(gone)[::-1]:
        arrs = _without_block(arrs, m)
    p = _image_parity(orc, arrs, 20.0, 5, 0.0, nu=1e9, mass_scale=1e25)
    assert p["steps_equal"] and p["max_pixel_rel_err"] <= 1e-8, p


def test_request_of_too_many_frequencies(cuda):
    """A request in device memory that names more than MK_MAX_NU frequencies
    (the Python layer refuses one) is rendered in the first MK_MAX_NU."""
    import ctypes
    from mahakala_gb300 import _lib
    from mahakala_gb300.grmhd.synthetic import make_synthetic_snapshot
    from mahakala_gb300.images import PreparedRender, RenderRequest
    arrs = make_synthetic_snapshot(nblocks=4, cells_per_block=8, extent=20., bhspin=0.94)
    nus = [86e9, 150e9, 230e9, 345e9]
    prep = PreparedRender([RenderRequest(_model(arrs), observing_frequency=nus, resolution=9, fov=20.0, **KW)])
    want = prep.launch()[0].clone()
    table = _lib.Request.from_buffer_copy(prep.table_bytes)
    for nnu in (_lib.MK_MAX_NU + 1, 1000):
        table.nnu = nnu
        prep.images[0].zero_()
        prep.reqs_dev.copy_(torch.frombuffer(bytearray(ctypes.string_at(ctypes.addressof(table), ctypes.sizeof(table))),
                                             dtype=torch.uint8))
        assert torch.equal(torch.nan_to_num(prep.launch()[0], nan=-1.0), torch.nan_to_num(want, nan=-1.0))


# a step over the horizon (here the rule stops this far above it) overflows
# floats before doubles; the fifth: more such rays than a block has room for;
# the last: its components are out of range, but finite
@pytest.mark.parametrize("spin,tol,div,half,res", [(-0.9, 1e-4, 40.0, 10.0, 48), (0.5, 1e-6, 40.0, 10.0, 48),
                                                   (0.5, 1e-8, 40.0, 10.0, 48), (0.94, 1e-8, 40.0, 10.0, 48),
                                                   (0.5, 1e-8, 10.0, 5.0, 200), (0.1, 1e-8, 20.0, 6.0, 64)])
def test_fp64_image_stop_reasons_at_the_horizon(cuda, orc, spin, tol, div, half, res):
    from mahakala_gb300.grmhd.synthetic import make_synthetic_snapshot
    from mahakala_gb300.images import RenderRequest, render_requests
    arrs = make_synthetic_snapshot(nblocks=2, cells_per_block=8, extent=20., bhspin=0.94)
    s0 = orc.initialize_geodesics_at_camera(spin, 60.0, 1000, -half, half, res)
    o = orc.integrate(s0, 4000, div, tol, spin)
    req = RenderRequest(_model(arrs), camera_inclination=60.0, fov=2 * half, resolution=res, bhspin=spin, tol=tol,
                        div=div, **dict(KW, max_nsteps=4000))
    render_requests([req], with_steps=True)
    steps, why = _np(req.out["nsteps"]).reshape(-1), _np(req.out["status"]).reshape(-1)
    # (which side of the horizon a last step lands on may turn on a rounding: 2 rays in 10^4)
    assert (steps != o["K"]).sum() + (why != o["why"]).sum() <= 2e-4 * len(s0)


# emission factors whose product leaves the floats' range, and is lifted into
# it again by the fit's polynomial; other images of this view differ from the
# oracle's by at most 3e-12 of a conditioned pixel
@pytest.mark.parametrize("u,mass", [(1e7, 1e22), (3e7, 1e22), (3e6, 1e22), (1e7, 3e21)])
def test_fp64_image_of_faint_factors(cuda, orc, u, mass):
    from mahakala_gb300.grmhd.synthetic import make_synthetic_snapshot
    arrs = make_synthetic_snapshot(nblocks=4, cells_per_block=8, extent=20., bhspin=0.94)
    arrs.uov[4] *= np.float32(u)
    p = _image_parity(orc, arrs, 20.0, 16, 0.94, nu=2e8, mass_scale=mass, r_high=1.)
    assert p["steps_equal"] and p["max_pixel_rel_err"] <= 1e-11, p


# beta to 1e15 and beyond beside an R_high of a million (its bar as above)
@pytest.mark.parametrize("u,B", [(1e7, 1e-4), (1e10, 1e-10), (1e9, 1e-6), (1e10, 1e-6)])
def test_fp64_image_of_large_beta(cuda, orc, u, B):
    from mahakala_gb300.grmhd.synthetic import make_synthetic_snapshot
    arrs = make_synthetic_snapshot(nblocks=4, cells_per_block=8, extent=20., bhspin=0.94)
    arrs.uov[4] *= np.float32(u)
    arrs.B *= np.float32(B)
    p = _image_parity(orc, arrs, 20.0, 16, 0.94, r_high=1e6)
    assert p["steps_equal"] and p["max_pixel_rel_err"] <= 1e-11, p


@pytest.mark.parametrize("r_high,r_low,gammas", [(1e6, 1e6, (1e6, 1e6)), (1e6, 1e-4, (1e6, 2. / 3)), (40., 1., (1e6, 1e6)),
                                                 (1e-4, 1e6, (1. / 3, 2. / 3)), (1e6, 1., (1. / 3, 2. / 3))])
def test_electrons_at_large_beta(cuda, r_high, r_low, gammas):
    """Against the formula in long double: 1e-15, five roundings (the binary64
    formula's largest error here is 9e-16)."""
    from mahakala_gb300.electrons import rlow_rhigh_model
    rng = np.random.default_rng(5)
    a = [10.0 ** rng.uniform(-100, 100, 20000), 10.0 ** rng.uniform(-100, 100, 20000), 10.0 ** rng.uniform(-9, 9.2, 20000)]
    t = _np(rlow_rhigh_model(*a, r_low=r_low, r_high=r_high, electron_gamma=1 + gammas[0], ion_gamma=1 + gammas[1]))
    dens, u, beta = (np.longdouble(x) for x in a)
    ge, gi = (np.longdouble((1 + g) - 1.0) for g in gammas)
    T = (r_high * beta * beta + r_low) / (1 + beta * beta)
    exact = np.longdouble(1.6726e-24) / np.longdouble(9.1094e-28) * u * ge * gi / (dens * (gi + ge * T))
    assert np.max(np.abs(t - exact) / exact) < 1e-15


# radii at which the fourth power of r, or its parts, leave the floats' range,
# and ones inside the ring
@pytest.mark.parametrize("spin", [0.0, 0.9])
def test_integrator_at_small_radii(cuda, orc, spin):
    from mahakala_gb300.geodesics import step_policy, trace
    x = np.array([0.3, 1e-2, 1e-4, 1e-6, 1e-9, 3e-10, 1e-11, 1e-13])
    s0 = np.zeros((len(x), 8))
    s0[:, 1], s0[:, 3] = x, 0.5 * x
    s0[:, 4:6] = 1.0
    with np.errstate(all="ignore"):
        o = orc.integrate(s0, 3, 1e4, 1e-4, spin, full=True)
    g = trace(s0, spin, step_policy(3, 1e4, 1e-4), rows=True)
    assert np.array_equal(_np(g["K"]), o["K"]) and np.array_equal(_np(g["why"]), o["why"])
    ok = o["K"] > 0
    assert np.max(rel_err(_np(g["dt"])[0][ok], o["dt"][0][ok])) < 1e-14


@pytest.mark.parametrize("case", range(5))
def test_captured_rays_as_exact_as_binary64(cuda, orc, case):
    """Captured rays' last wavevectors against an integration in long double
    (golden/make_wide.py): the geometric mean of 40 rays' errors at most 1.5
    times that of the oracle's binary64 (rounding scatters each error by a
    factor of 3 or so, a mean of 40 by 1.2)."""
    from conftest import golden
    from mahakala_gb300.geodesics import step_policy, trace
    d = golden("wide")
    s0, K, hi, lo = (d[f"{k}_{case}"] for k in ("s0", "K", "hi", "lo"))
    spin, tol = float(d[f"spin_{case}"]), float(d[f"tol_{case}"])
    g = trace(s0, spin, step_policy(4000, 40.0, tol))
    assert np.array_equal(_np(g["K"]), K)

    def mean_error(x):
        e = np.linalg.norm(((x - hi) - lo)[:, 4:], axis=1) / np.linalg.norm(hi[:, 4:], axis=1)
        return np.exp(np.mean(np.log(e)))

    ours, theirs = mean_error(_np(g["state"])), mean_error(orc.integrate(s0, 4000, 40.0, tol, spin)["state"])
    assert ours <= 1.5 * theirs, (ours, theirs)


@pytest.mark.parametrize("case", [3, 4])
def test_shadow_radii_as_exact_as_binary64(cuda, orc, case):
    """Radii at the horizon of select_photons_integrator against long double
    (golden/make_wide.py): the median error at most twice 3e-16 + that of the
    binary64 radii r (the spacing of doubles at r, over sqrt(12), and 7e-16 and
    4e-15 measured of a binary64 integration at spins 0.94 and 0.998)."""
    from conftest import golden
    from mahakala_gb300.geodesics import select_photons_integrator
    d = golden("wide")
    r = select_photons_integrator(60.0, d[f"angle_{case}"], d[f"radius_{case}"], float(d[f"spin_{case}"]))
    hi, lo = d[f"r_hi_{case}"], d[f"r_lo_{case}"]
    assert len(r) > 100
    assert np.median(np.abs((r - hi) - lo) / hi) <= {3: 2 * 1e-15, 4: 2 * 4.3e-15}[case]


@pytest.mark.parametrize("case", range(8))
def test_escaped_rays_as_exact_as_binary64(cuda, orc, case):
    """Escaped rays under step rules of long and short steps, from afar and
    near by, against long double (golden/make_wide.py): the geometric mean of
    up to 100 rays' errors at most 1.5 times the oracle's, as above."""
    from conftest import golden
    from mahakala_gb300.geodesics import step_policy, trace
    d = golden("wide")
    s0, K, hi, lo = (d[f"rule_{k}_{case}"] for k in ("s0", "K", "hi", "lo"))
    spin, value = float(d[f"rule_spin_{case}"]), float(d[f"rule_value_{case}"])
    if str(d[f"rule_{case}"]) == "div":
        g = trace(s0, spin, step_policy(4000, value, 1e-4))
        o = orc.integrate(s0, 4000, value, 1e-4, spin)
    else:
        g = trace(s0, spin, step_policy(4000, kind="fixed", hfrac=value))
        o = orc.trace_fixed(s0, 4000, spin, hfrac=value)
    assert len(s0) > 60 and np.array_equal(_np(g["K"]), K)

    def mean_error(x):
        x, r = ((v * (1, 1, 1, 10, 10, 10, 10)) for v in (((x - hi) - lo)[:, 1:], hi[:, 1:]))
        return np.exp(np.mean(np.log(np.maximum(np.linalg.norm(x, axis=1) / np.linalg.norm(r, axis=1), 1e-18))))

    ours, theirs = mean_error(_np(g["state"])), mean_error(o["state"])
    assert ours <= 1.5 * theirs, (ours, theirs)
