"""The line elements' shorter forms where they are chosen: maps with and without entries outside the plane blocks
(single entries of every kind among them), crab cavities of one to eight harmonics, boosts of either sign and of a large
angle, each with particles that are not finite among the others; float64 within 1e-13 of each component's RMS of the
oracle (test_gpu_line.py's bound), and the same particles non-finite."""
import numpy as np
import pytest

from helpers import beams
from test_gpu_line import assert_close, gpu_track, oracle_track

pytestmark = pytest.mark.gpu


def _check(elems, turns=2):
    e, _ = beams(20_001, 16)
    good = e.copy()
    assert_close(gpu_track(elems, good.copy(), turns=turns), oracle_track(elems, good.copy(), turns=turns))
    for k, bad in enumerate((np.nan, np.inf, -np.inf)):
        for c in range(6):
            e[c, 100 * c + k] = bad
    got, want = gpu_track(elems, e.copy(), turns=turns), oracle_track(elems, e.copy(), turns=turns)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    both = np.isfinite(want).all(axis=0)
    assert_close(got[:, both], want[:, both])


# a planar map, and maps whose only entries outside the plane blocks are one dispersion, one coupling or one crab term's
MAPS = [{}, dict(eta1=(0.2, 0.0, 0.0, 0.0)), dict(eta2=(0.0, 0.0, 0.0, 1e-3)), dict(R1=(0.0, 0.02, 0.0, 0.0)),
        dict(zeta1=(0.0, -1e-3, 0.0, 0.0))]


@pytest.mark.parametrize("kw", MAPS)
def test_maps_with_and_without_coupling(kw):
    from octo_b200 import line as ln
    _check([ln.Linear6DSpec(beta1=(0.7, 0.05, 12.0), alpha1=(0.1, -0.2, 0.0), dmu=(0.3, -1.1, 0.02), **kw)])


@pytest.mark.parametrize("n", [1, 2, 5, 6, 7, 8])
def test_crab_harmonics(n):
    from octo_b200 import line as ln
    sx = tuple(0.01 / (h + 1) for h in range(n))
    sy = tuple(0.002 * (h % 2) for h in range(n))
    _check([ln.ThinCrabCavitySpec(197e6, N=n, strengthX=sx, strengthY=sy, phase=tuple(0.1 * h for h in range(n)))])


@pytest.mark.parametrize("angle", [0.0, 12.5e-3, -0.4, 1.2])
def test_boost_pair(angle):
    from octo_b200 import line as ln
    _check([ln.LorentzBoostSpec(angle)], turns=1)
    _check([ln.RevLorentzBoostSpec(angle)], turns=1)


def _same(elems, c):
    """Finite and infinite values where the oracle has them, of the oracle's values."""
    got, want = gpu_track(elems, c.copy(), turns=1), oracle_track(elems, c.copy(), turns=1)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    there = ~np.isnan(want)
    assert np.array_equal(np.isinf(got), np.isinf(want)) and np.array_equal(np.sign(got[there]), np.sign(want[there]))
    there &= ~np.isinf(want)
    np.testing.assert_allclose(got[there], want[there], rtol=1e-14, atol=0)  # a few roundings of each side


@pytest.mark.parametrize("angle", [1.2, -0.4])
def test_boost_quotients_that_overflow(angle):
    from octo_b200 import line as ln
    c = np.zeros((6, 8))
    c[3] = [1.7e308, -1.7e308, 1e-310, 0.0, 5e-324, -1e-300, 1e-3, 1e3]
    c[4] = [0.0, 1e-3, 1.7e308, -1.7e308, 1e-320, 1e300, 0.0, -0.0]
    _same([ln.LorentzBoostSpec(angle)], c)


@pytest.mark.parametrize("f,strength", [(1.0, 1.6e308), (1e-303, 1e-310), (1e-303, 1e-3), (1e300, 1e-3)])
def test_crab_quotients_that_overflow(f, strength):
    from octo_b200 import line as ln
    c = np.zeros((6, 3))
    c[0], c[4] = [1e-4, 0.0, -1e-4], [1e-2, 0.0, -3e-2]
    if f == 1e300:
        c[4] = 0.0  # the phase alone: no reduction of a huge angle
    _same([ln.ThinCrabCavitySpec(f, N=2, strengthX=(strength, strength), strengthY=(0.0, -strength), phase=(1.0, -0.5))], c)
