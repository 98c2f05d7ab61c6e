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
