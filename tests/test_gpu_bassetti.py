"""The Bassetti-Erskine response of the soft-Gaussian kick where its evaluation changes: the round closed form, the
near-round series, the blend, the elliptic form just above it and at strong aspect ratios with either axis the long
one; each at points on the axes, inside and outside the radial series' region, in the rational approximation's region
and in the far region of w(z).  One pair of single slices, kbb = 1, so a probe's momentum is the kick itself."""
import numpy as np
import pytest

from helpers import oracle_params, E_PARAMS, P_PARAMS
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _source(n, sx, sy):
    rng = np.random.default_rng(5)
    u = rng.standard_normal(n)
    u = (u - u.mean()) / u.std()
    c = np.zeros((6, n))
    c[0], c[2] = sx * u, sy * u[rng.permutation(n)]  # the same values: the sample's sigma ratio is sx / sy
    return c


def _probes(sx, sy, n):
    a = np.array([0.0, 1e-3, 5e-3, 7e-3, 2e-2, 0.3, 1.0, 3.0, 6.5, 15.0, 60.0])
    a = np.concatenate([a, -a[1:]])
    gx, gy = np.meshgrid(a, a)
    c = np.zeros((6, n))
    c[0], c[2] = sx * np.resize(gx.ravel(), n), sy * np.resize(gy.ravel(), n)
    return c


def _collide(e, p):
    """Luminosity and the probes' coordinates of one pair of single slices, here and (in place) in the oracle."""
    import octo_b200 as ob
    solver = ob.GaussianPoissonSolver(slicing=ob.LongitudinalSlicing(nslices=1, method="normal_quantile"), kbb1=1.0,
                                      kbb2=1.0, luminosity_scale=1.0, gaussian_when_luminosity=1)
    params = [ob.BeamParams(q["charge"], q["mass"], q["energy"], q["r0"], q["npart"]) for q in (E_PARAMS, P_PARAMS)]
    be, bp = ob.Beam.from_numpy(e, params[0]), ob.Beam.from_numpy(p, params[1])
    lum = ob.collide(solver, be, bp)
    opt = orc.OracleOptions(nslices1=1, nslices2=1, kbb1=1.0, kbb2=1.0, luminosity_scale=1.0)
    ref = orc.gaussian_collide(opt, e, p, *oracle_params(), 0.0, 1, False, False, "hirata", False)
    return lum, ref, bp.numpy()


@pytest.mark.parametrize("aspect", [1.0, 1.0 + 1e-4, 1.0 + 3e-4, 1.0 + 5e-4, 1.02, 11.0, 1.0 / 11.0, 150.0])
@pytest.mark.parametrize("n", [441, 3 * 444 * 256 + 77])  # one particle a thread; several, with a ragged last block
def test_kick_of_every_regime(aspect, n):
    sy = 1e-5
    e, p = _source(4001, aspect * sy, sy), _probes(aspect * sy, sy, n)
    lum, ref, got = _collide(e, p)
    assert abs(lum / ref - 1.0) < 1e-12
    # each side rounds w(z) to about 4 x 1.1e-16, and the elliptic form multiplies the difference of two such values by
    # 2 sqrt(pi) / (sqrt(2) sqrt(2 eta) sigma) <= 84 / sigma (eta >= 4.4e-4), where the largest kick is 0.45 / sigma:
    # 2 x 4.4e-16 x 84 / 0.45 = 1.6e-13 of it; the bound is twice that
    for k in (1, 3):
        assert np.max(np.abs(got[k] - p[k])) <= 3e-13 * np.max(np.abs(p[[1, 3]]))
    # the longitudinal kick here is the drift term of the kicked momenta alone
    assert np.max(np.abs(got[5] - p[5])) <= 2e-12 * np.max(np.abs(p[5])) + 1e-16


@pytest.mark.parametrize("aspect", [1.0, 1.0 + 5e-4, 1.02, 11.0, 1.0 / 11.0, 150.0])
def test_hessians_of_every_regime(aspect):
    """A source whose momenta are correlated with its positions: the longitudinal kick then holds both Hessians."""
    sy = 1e-5
    e, p = _source(4001, aspect * sy, sy), _probes(aspect * sy, sy, 441)
    e[1], e[3] = 3.0 * e[0], -2.0 * e[2]  # au = 2 cov(x, px) = 6 sigma_x^2, du = -4 sigma_y^2 at zero drift
    lum, ref, got = _collide(e, p)
    assert abs(lum / ref - 1.0) < 1e-12
    # The momenta as in test_kick_of_every_regime, and with their error dK, 2 x 4.4e-16 x 2.51 / sqrt(q^2 - 1) over the
    # short sigma (q the aspect ratio, at most 84 in its place near round): a Hessian is (x Kx + y Ky - 2 (1 - ..)) over the
    # difference of the variances, so over some three sigma its error is 3 (q + 1) dK / (q^2 - 1) in units of 1 / short^2,
    # and never less than a few roundings of its largest term; times a quarter of au, 6 q^2 / 4 long variances.
    q = max(aspect, 1.0 / aspect)
    amp = min(2.51 / np.sqrt(max(q * q - 1.0, 1e-9)), 84.0)
    dk = 2 * 4.4e-16 * amp
    dh = 3.0 * (q + 1.0) * dk / max(q * q - 1.0, 8.8e-4) + 1e-14 / (q * q)
    bound = 2.0 * 1.5 * q * q * dh
    assert np.max(np.abs(got[5] - p[5])) <= bound + 1e-14 * np.max(np.abs(p[5])), (np.max(np.abs(got[5] - p[5])), bound)
    assert np.max(np.abs(p[5])) > 0.5  # the Hessian terms are there


@pytest.mark.parametrize("aspect", [11.0, 1.0 / 11.0, 150.0])
def test_particles_far_outside(aspect):
    """Coordinates whose square over the variance overflows: no density, and the kick of a distant charge."""
    sy = 1e-5
    e, p = _source(4001, aspect * sy, sy), _probes(aspect * sy, sy, 441)
    p[0, 7], p[2, 9], p[0, 11], p[2, 11] = 1e153, -1e153, -3e152, 2e151
    lum, ref, got = _collide(e, p)
    assert np.isfinite(ref) and abs(lum / ref - 1.0) < 1e-12
    far = [7, 9, 11]
    assert np.isfinite(got).all() and np.isfinite(p).all()
    np.testing.assert_allclose(got[:, far], p[:, far], rtol=1e-13, atol=1e-300)
