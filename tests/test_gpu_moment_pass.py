"""The one-pass moment rows where a pivot instead of the mean could lose something: beams of a few particles, sorted
ones, one stray particle, a centre far from zero, equal coordinates, sizes around the pivot's 4096 samples and the
grid's last threads."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _beam(kind, n):
    rng = np.random.default_rng(n)
    c = rng.standard_normal((6, n)) * np.array([1e-4, 2e-4, 1e-5, 2e-4, 6e-2, 6e-4])[:, None]
    if kind == "sorted":
        c.sort(axis=1)
    elif kind == "stray":
        c[0, n // 2] = 1e3
        c[5, n - 1] = -40.0
    elif kind == "offset":
        c += np.array([1.0, -3.0, 2.0, 0.5, 1e3, -1.0])[:, None]
    elif kind == "equal":
        c[2] = 0.1
        c[4] = -7e-3
    return c


@pytest.mark.parametrize("kind", ["plain", "sorted", "stray", "offset", "equal"])
@pytest.mark.parametrize("n", [1, 2, 33, 4095, 4096, 4097, 592 * 256 - 1, 2 * 592 * 256 + 1, 400_003])
def test_row_matches_extended_precision(kind, n):
    import octo_b200 as ob
    c = _beam(kind, n)
    obs = ob.MomentObserver("b", orders=(1, 2))
    obs.observe(3, ob.Beam.from_numpy(c, ob.BeamParams(1.0, 1.0, 1.0, 1.0, 1.0)))
    row = obs.rows()[0]
    w = c.astype(np.longdouble)
    mean = w.mean(axis=1)
    d = w - mean[:, None]
    rms = np.sqrt((d * d).mean(axis=1))
    assert row[0] == 3.0
    # every partial sum is of at most a few thousand terms before the folds: 1e-13 of the moment's natural scale
    # covers their rounding; a mean is off by its own rounding as well
    np.testing.assert_array_less(np.abs(row[1:7] - mean), 1e-13 * rms + 2.3e-16 * np.abs(mean) + 1e-300)
    k = 7
    for i in range(6):
        for j in range(i, 6):
            want = (d[i] * d[j]).mean()
            # the extended-precision mean is itself off by up to 1e-16 of its value
            own = 1e-32 * abs(mean[i] * mean[j])
            assert abs(row[k] - want) <= 1e-13 * rms[i] * rms[j] + own + 1e-300, (i, j, row[k], want)
            k += 1


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_samples_leave_the_pivot(bad):
    import octo_b200 as ob
    n = 32_768
    c = _beam("plain", n)
    c[1, ::8] = bad  # every sampled particle
    params = ob.BeamParams(1.0, 1.0, 1.0, 1.0, 1.0)
    rows = {}
    for mask in (False, True):
        obs = ob.MomentObserver("b", orders=(1, 2), mask_lost=mask)
        obs.observe(0, ob.Beam.from_numpy(c, params))
        rows[mask] = obs.rows()[0]
    live = c[:, np.isfinite(c[1])]
    np.testing.assert_allclose(rows[True][1:7], live.mean(axis=1), rtol=0, atol=1e-17)
    names = obs.column_names
    for k, name in enumerate(names):
        if k and name[2] != "0":  # a moment of px: its mean keeps the sum's value, the central ones are NaN
            assert np.isnan(rows[False][k]) if sum(map(int, name[1:])) == 2 else not np.isfinite(rows[False][k])
        else:
            assert np.isfinite(rows[False][k])
    torch.cuda.synchronize()


def _live_row(c, dtype):
    """Row of a masked observer and the extended-precision moments of its live particles."""
    import octo_b200 as ob
    c = c.astype(np.float32).astype(np.float64) if dtype == torch.float32 else c
    obs = ob.MomentObserver("b", orders=(1, 2), mask_lost=True)
    obs.observe(0, ob.Beam.from_numpy(c, ob.BeamParams(1.0, 1.0, 1.0, 1.0, 1.0), dtype=dtype))
    return obs.rows()[0], np.ascontiguousarray(c[:, np.isfinite(c).all(axis=0)], dtype=np.longdouble)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("far", [1e4, 1e10])
@pytest.mark.parametrize("case", ["one in twenty", "every sample", "three left", "one left"])
def test_lost_particles_leave_the_pivot(case, far, dtype):
    """A lost particle (one coordinate NaN or infinite) may hold any finite values in the others: they are no part of a
    masked row, so they must not move the pivot away from the live particles either."""
    n = 200_000
    c = _beam("plain" if case == "one in twenty" else "offset", n)
    lost = {"one in twenty": np.arange(0, n, 20), "every sample": np.arange(n)[np.arange(n) % 17 != 5],
            "three left": np.setdiff1d(np.arange(n), [77_777, 77_779, 150_000]),
            "one left": np.setdiff1d(np.arange(n), [199_999])}[case]
    c[:, lost] = far
    c[3, lost] = np.nan
    c[3, lost[::2]] = np.inf
    row, live = _live_row(c, dtype)
    mean = live.mean(axis=1)
    d = live - mean[:, None]
    rms = np.sqrt((d * d).mean(axis=1))
    # the bounds of test_row_matches_extended_precision
    np.testing.assert_array_less(np.abs(row[1:7] - mean), 1e-13 * rms + 2.3e-16 * np.abs(mean) + 1e-300)
    k = 7
    for i in range(6):
        for j in range(i, 6):
            own = 1e-32 * abs(mean[i] * mean[j])
            assert abs(row[k] - (d[i] * d[j]).mean()) <= 1e-13 * rms[i] * rms[j] + own + 1e-300, (i, j, row[k])
            k += 1


@pytest.mark.parametrize("kind", ["plain", "sorted", "stray", "offset", "equal", "lost"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 4097, 592 * 256 + 1, 400_003])
def test_rows_without_second_moments(n, dtype, kind):
    """Rows of order 1, and of 1 and 3, sum the deviations without their products, about a pivot of their own."""
    import octo_b200 as ob
    c = _beam("offset" if kind == "lost" else kind, n)
    if kind == "lost":
        c[:, 1::3] = 1e6
        c[2, 1::3] = np.nan
    if dtype == torch.float32:
        c = c.astype(np.float32).astype(np.float64)
    live = np.ascontiguousarray(c[:, np.isfinite(c).all(axis=0)], dtype=np.longdouble)  # rows of pairwise sums
    mean = live.mean(axis=1)
    d = live - mean[:, None]
    rms = np.sqrt((d * d).mean(axis=1))
    for orders in ((1,), (1, 3)):
        obs = ob.MomentObserver("b", orders=orders, mask_lost=kind == "lost")
        obs.observe(4, ob.Beam.from_numpy(c, ob.BeamParams(1.0, 1.0, 1.0, 1.0, 1.0), dtype=dtype))
        row = dict(zip(obs.column_names, obs.rows()[0]))
        got = np.array([row["m" + "0" * k + "1" + "0" * (5 - k)] for k in range(6)])
        # the bounds of test_row_matches_extended_precision
        np.testing.assert_array_less(np.abs(got - mean), 1e-13 * rms + 2.3e-16 * np.abs(mean) + 1e-300)
        if 3 in orders:
            for k in range(6):
                third = (d[k] ** 3).mean()
                assert abs(row["m" + "0" * k + "3" + "0" * (5 - k)] - third) <= 1e-12 * max(rms[k] ** 3, (abs(d[k]) ** 3).mean()) \
                    + 1e-15 * abs(mean[k]) * rms[k] ** 2 + 1e-300
