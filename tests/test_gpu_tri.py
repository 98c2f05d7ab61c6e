"""The paths on the FP32 pipe (float pairs and triples) where their rules and
edges lie: small and ragged launches of the FP64 render, requests and samples
it leaves to binary64, the integrators at few rays and out of range, rows
frozen apart, the stage kernels over wide ranges and at block faces, and the
several-bisections-a-pass shadow.  Against the oracle at the bars of the other
tests (FP64 images 1e-8 a conditioned pixel, fluid scalars 1e-12, synchrotron
1e-11), or bit for bit against the general path where each ray's arithmetic
is the same.
"""

import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu

KW = dict(mass_scale=3e26, M_bh=6.5e9 * 1.989e33, r_high=40, max_nsteps=3000)


def _np(t):
    return t.detach().cpu().numpy()


def _snapshot(seed=11):
    from mahakala_gb300.grmhd.synthetic import make_synthetic_snapshot
    return make_synthetic_snapshot(nblocks=4, cells_per_block=16, extent=50.0, bhspin=0.94, seed=seed)


def _multilevel():
    from mahakala_gb300.grmhd.synthetic import make_multilevel_snapshot
    return make_multilevel_snapshot(nblocks=4, cells_per_block=8, extent=20., bhspin=0.94,
                                    refine=[(0, 1, 1, 1), (0, 2, 2, 2), (1, 2, 2, 2)])


def _model(arrs):
    from mahakala_gb300.grmhd.athenak import AthenakFluidModel
    return AthenakFluidModel(arrs, arrs.bhspin, fluid_gamma=13. / 9)


@pytest.fixture(scope="module")
def medium():
    return _snapshot()


def _parity(orc, arrs, img, steps, fov, res, nu, inc=60.0, **kw):
    osnap = orc.OracleSnapshot(arrs)
    s0 = orc.initialize_geodesics_at_camera(arrs.bhspin, inc, 1000, -fov / 2, fov / 2, res)
    kw = dict(kw or KW, observing_frequency=nu)
    ref, rsteps = orc.render_rays(osnap, s0, **kw)
    pert, psteps = orc.render_rays(osnap, orc.perturbed(s0), **kw)
    return orc.image_parity(img.reshape(len(np.atleast_1d(nu)), -1), steps, ref, rsteps, pert, psteps)


# 4 rays: one a warp; 36: a ragged spread over the couples; 4900 and 22801:
# some and all warps filled, the last ones in part
@pytest.mark.parametrize("res,nu", [(2, 230e9), (6, [86e9, 230e9, 345e9, 690e9]), (70, [86e9, 230e9]), (151, 230e9)])
def test_fp64_image_sizes(cuda, orc, medium, res, nu):
    from mahakala_gb300.images import RenderRequest, render_requests
    req = RenderRequest(_model(medium), camera_inclination=60.0, fov=40.0, resolution=res, observing_frequency=nu, **KW)
    img = _np(render_requests([req], with_steps=True)[0])
    req.out["check"]()
    p = _parity(orc, medium, img, _np(req.out["nsteps"]), 40.0, res, nu)
    assert p["steps_equal"] and p["max_pixel_rel_err"] <= 1e-8 and p["flux_rel_err"] <= 1e-8, p


# the same image from primitives of other sizes (mass_scale takes the factor
# back), and blocks whose primitives lie at and below the smallest floats:
# rescaled samples, or samples and requests taken in binary64
@pytest.mark.parametrize("where,f", [("all", 1e-6), ("all", 1e-12), ("all", 1e-24), ("all", 1e12), ("half", 1e-28),
                                     ("half", 1e-36)])
def test_fp64_image_of_extreme_primitives(cuda, orc, where, f):
    from mahakala_gb300.images import RenderRequest, render_requests
    arrs = _snapshot(5)
    at = slice(None) if where == "all" else slice(None, None, 2)
    arrs.uov[0, at] *= np.float32(f)
    arrs.uov[4, at] *= np.float32(f)
    arrs.B[:, at] *= np.float32(f ** 0.5)
    kw = dict(KW, mass_scale=3e26 / (f if where == "all" else 1.0))
    req = RenderRequest(_model(arrs), camera_inclination=60.0, fov=40.0, resolution=20, **kw)
    img = _np(render_requests([req], with_steps=True)[0])
    p = _parity(orc, arrs, img, _np(req.out["nsteps"]), 40.0, 20, 230e9, **kw)
    assert p["steps_equal"] and p["max_pixel_rel_err"] <= 1e-8, p


def test_fp64_image_of_refined_blocks(cuda, orc):
    from mahakala_gb300.images import RenderRequest, render_requests
    arrs = _multilevel()
    req = RenderRequest(_model(arrs), camera_inclination=60.0, fov=20.0, resolution=24, **KW)
    img = _np(render_requests([req], with_steps=True)[0])
    p = _parity(orc, arrs, img, _np(req.out["nsteps"]), 20.0, 24, 230e9)
    assert p["steps_equal"] and p["max_pixel_rel_err"] <= 1e-8, p


def test_requests_outside_the_pairs_range_beside_others(cuda, medium):
    """Requests the float pairs cannot hold (here an L_unit above 1e20) go to the binary64 kernel, the rest of a job of 130 requests do not,
    and each gives what it gives alone."""
    from mahakala_gb300.images import RenderRequest, render_requests
    m = _model(medium)

    def req(i):
        kw = dict(KW, mass_scale=1e26 * (1 + i % 5), camera_inclination=20.0 + i, fov=40.0, resolution=3 + i % 4)
        if i % 40 == 7:
            kw["M_bh"] = 1e50
        return RenderRequest(m, **kw)

    together = render_requests([req(i) for i in range(130)])
    for i in (0, 6, 7, 8, 47, 87, 127, 128, 129):
        alone = render_requests([req(i)])[0]
        assert torch.equal(torch.nan_to_num(together[i], nan=-1.0), torch.nan_to_num(alone, nan=-1.0)), i


@pytest.mark.parametrize("n", [1, 31, 33, 1217])
@pytest.mark.parametrize("kind", ["reference", "fixed"])
def test_integrators_at_few_rays(cuda, orc, n, kind):
    from mahakala_gb300.geodesics import step_policy, trace
    from test_gpu_vacuum import check_end_states
    a = 0.5
    s0 = orc.initialize_geodesics_at_camera(a, 60, 1000, -10, 10, 36)[:n]
    run = ((lambda s: orc.integrate(s, 2000, 40.0, 1e-4, a)) if kind == "reference" else
           (lambda s: orc.trace_fixed(s, 2000, a)))
    o, amp = orc.conditioning(run, s0, **({} if kind == "reference" else dict(key_steps="nsteps")))
    g = trace(s0, a, step_policy(2000, 40.0, 1e-4, kind=kind))
    assert np.array_equal(_np(g["why"]), o["why"])
    check_end_states(orc, _np(g["K"]), _np(g["state"]), o["K" if kind == "reference" else "nsteps"], o["state"], amp,
                     f"{kind}, {n} rays")


def test_integrator_keeps_given_doubles(cuda):
    """Row 0, and the end state of a run of no steps, are the given bits,
    whatever they hold (triples are taken up by bit operations)."""
    from mahakala_gb300.geodesics import step_policy, trace
    rng = np.random.default_rng(2)
    s0 = rng.normal(size=(257, 8)) * 10.0 ** rng.uniform(-3, 3, (257, 8))
    odd = [0.0, -0.0, 5e-324, -1e-310, 1e-40, 2.0 ** -76, 2.0 ** 105, -2.0 ** 104.99, 1e39, 1e300, np.inf, -np.inf]
    for i, v in enumerate(odd):
        s0[10 + i, i % 8] = v
    g = trace(s0, 0.9, step_policy(0))
    assert np.array_equal(_np(g["state"]).view(np.int64), s0.view(np.int64))
    g = trace(s0, 0.9, step_policy(1, 40.0, 1e-4), rows=True)
    assert np.array_equal(_np(g["S"][0]).view(np.int64), s0.view(np.int64))


# wavevectors and radii past the triples' range are integrated in binary64
@pytest.mark.parametrize("kscale,xscale,stops_at", [(1e-3, 1.0, 60), (1e-30, 1.0, 60), (1e13, 1.0, 0), (1.0, 1e9, 0)])
def test_integrator_out_of_range(cuda, orc, kscale, xscale, stops_at):
    from mahakala_gb300.geodesics import step_policy, trace
    a = 0.5
    s0 = orc.initialize_geodesics_at_camera(a, 60, 1000, -10, 10, 6)
    s0[:, 4:] *= kscale
    s0[:, 1:4] *= xscale
    with np.errstate(all="ignore"):
        o = orc.integrate(s0, 60, 40.0, 1e-4, a)
    assert (o["K"] == stops_at).all()
    g = trace(s0, a, step_policy(60, 40.0, 1e-4))
    assert np.array_equal(_np(g["K"]), o["K"]) and np.array_equal(_np(g["why"]), o["why"])
    st = _np(g["state"])
    # against each vector's own norm: 60 steps far from the hole amplify nothing
    for sl in (slice(0, 4), slice(4, 8)):
        x, r = st[:, sl], o["state"][:, sl]
        assert np.max(np.linalg.norm(x - r, axis=1) / np.linalg.norm(r, axis=1)) < 1e-10


@pytest.mark.parametrize("n,N", [(1, 40), (36, 700), (36, 3000), (144, 1)])
def test_frozen_rows_apart(cuda, orc, n, N):
    """geodesic_integrator's rows, frozen after the trim, are the rows one
    mk_integrate with rows writes."""
    import mahakala_gb300 as mk
    from mahakala_gb300.geodesics import step_policy, trace, trimmed_rows
    s0 = orc.initialize_geodesics_at_camera(0.5, 60, 1000, -10, 10, 12)[:n]
    S, dt = mk.geodesic_integrator(N, s0, 40.0, 1e-2, 0.5)
    r = trace(s0, 0.5, step_policy(N, 40.0, 1e-2), rows=True)
    nt = trimmed_rows(r["K"], N)
    assert S.shape[0] == nt
    assert torch.equal(S, r["S"][:nt]) and torch.equal(dt, r["dt"][:nt])


@pytest.mark.parametrize("error_allowed,max_it,n", [(1e-3, 40, 7), (1e-3, 5, 7), (0.3, 40, 1), (1e-3, 40, 300)])
def test_shadow_passes_of_any_depth(cuda, monkeypatch, error_allowed, max_it, n):
    """Several bisections a pass give the radii of one a pass."""
    from mahakala_gb300 import geodesics as g
    ang = np.linspace(0.0, 2 * np.pi, n, endpoint=False)
    kw = dict(error_allowed=error_allowed, max_it=max_it)
    many = g.find_shadow_bisection_angles(0.7, 60.0, ang, **kw)
    monkeypatch.setattr(g, "SHADOW_RAYS", 1)
    assert np.array_equal(many, g.find_shadow_bisection_angles(0.7, 60.0, ang, **kw))


def test_electrons_over_wide_ranges(cuda, orc):
    """1e-300 .. 1e300 and zeros, infinities and NaN: 2e-15, eight roundings
    of the oracle's own evaluation."""
    from mahakala_gb300.electrons import rlow_rhigh_model
    rng = np.random.default_rng(0)
    odd = np.array([0.0, -0.0, 1e-300, 1e300, 5e-324, np.inf, np.nan, -1.0, 1.0])
    for scale in (3.0, 30.0, 150.0):
        a = 10.0 ** rng.uniform(-scale, scale, (3, 4000))
        for i in range(3):
            a[i, rng.integers(0, 4000, 60)] = rng.choice(odd, 60)
        with np.errstate(all="ignore"):
            ref = orc.rlow_rhigh_model(*a, r_low=1.0, r_high=40.0)
        t = _np(rlow_rhigh_model(*a, r_low=1.0, r_high=40.0))
        assert np.array_equal(np.isnan(t), np.isnan(ref)) and np.array_equal(np.isinf(t), np.isinf(ref))
        ok = np.isfinite(ref) & (np.abs(ref) > 1e-290)
        assert np.max(rel_err(t[ok], ref[ok])) < 2e-15


@pytest.mark.parametrize("invariant", [True, False])
def test_synchrotron_over_wide_ranges(cuda, orc, invariant):
    import mahakala_gb300 as mk
    rng = np.random.default_rng(1)
    n = 20000
    args = [10.0 ** rng.uniform(-5, 12, n), 10.0 ** rng.uniform(-3, 4, n), 10.0 ** rng.uniform(-6, 4, n),
            np.arccos(rng.uniform(-1, 1, n)), 10.0 ** rng.uniform(8, 14, n)]
    odd = np.array([0.0, -0.0, 1e-300, 1e300, 5e-324, np.inf, np.nan, -1.0])
    for a in args:
        a[rng.integers(0, n, 100)] = rng.choice(odd, 100)
    args[3][:4] = (0.0, np.pi, 1e-12, np.pi / 2)
    kw = dict(invariant=invariant, rescale_nu=1 / 230e9)
    with np.errstate(all="ignore"):
        refs = orc.synchrotron_coefficients(*args, **kw)
    for x, ref in zip(mk.synchrotron_coefficients(*args, **kw), refs):
        x = _np(x)
        assert np.array_equal(np.isnan(x), np.isnan(ref)) and np.array_equal(np.isinf(x), np.isinf(ref))
        ok = np.isfinite(ref) & (np.abs(ref) > 1e-290)
        assert np.max(rel_err(x[ok], ref[ok])) < 1e-11


@pytest.mark.parametrize("refined", [False, True])
def test_fluid_at_faces_and_edges(cuda, orc, refined):
    """Points on block faces, cell centres and one ulp beside them, at the
    mesh's edge and off it, and wavevectors of any size."""
    from mahakala_gb300.grmhd.synthetic import make_synthetic_snapshot
    arrs = _multilevel() if refined else make_synthetic_snapshot(nblocks=4, cells_per_block=8, extent=20., bhspin=0.94)
    rng = np.random.default_rng(3)
    at = np.concatenate([np.linspace(-20, 20, 5), np.linspace(-20, 20, 65), np.nextafter([10, 10, -20, 20, 20],
                                                                                        [0, 20, 0, 30, 0]),
                         [-0.0, 0.0, 1e-30, 25., -25., 1e5]])
    X = rng.choice(at, (6000, 3))
    X[:3000, 1] = rng.uniform(-22, 22, 3000)
    X[1000:4000, 2] = rng.uniform(-22, 22, 3000)
    X = X[(X ** 2).sum(axis=1) > 4.0]
    K = rng.normal(size=(len(X), 4))
    K[:50] *= 1e13
    K[50:100] *= 1e-13
    S = np.concatenate([np.zeros((len(X), 1)), X, K], 1)
    ref = orc.OracleSnapshot(arrs).get_fluid_scalars_from_geodesics(S)
    g = _model(arrs).get_fluid_scalars_from_geodesics(S)
    # k.u is a sum of terms of the size of k^2-free |k|: a random K can cancel in it
    kn = np.linalg.norm(K, axis=1)
    for k in ("dens", "u", "b"):
        x = _np(g[k])
        assert np.array_equal(np.isnan(x), np.isnan(ref[k])), k
        assert np.nanmax(rel_err(x, ref[k])) < 1e-12, k
    x = _np(g["kdotu"])
    assert np.array_equal(np.isnan(x), np.isnan(ref["kdotu"]))
    assert np.nanmax(np.abs(x - ref["kdotu"]) / np.maximum(np.abs(ref["kdotu"]), kn)) < 1e-12


@pytest.mark.parametrize("nsteps,npx", [(2, 1), (16, 65), (17, 64), (18, 63), (34, 1), (150, 129), (6, 40000),
                                        (14, 40001), (20, 38912)])
def test_transfer_read_ahead(cuda, orc, nsteps, npx):
    """Rows read 16 ahead, or 6 for many pixels, 64 pixels a block: each side
    of each."""
    import mahakala_gb300 as mk
    rng = np.random.default_rng(nsteps)
    em, ab = rng.uniform(0, 1e-3, (2, nsteps, npx))
    dt = -rng.uniform(0.1, 1.0, (nsteps, npx))
    ref = orc.solve_specific_intensity(em, ab, dt, 10.0)
    assert np.max(rel_err(_np(mk.solve_specific_intensity(em, ab, dt, 10.0)), ref)) < 1e-13
