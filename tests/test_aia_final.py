"""The phase that AIA returns for given shifts (no iteration): any first shift,
pixels whose frames are not finite, against plain numpy in 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(m, h, w, deltas, seed=0):
    rng = np.random.default_rng(seed)
    phi = rng.uniform(-np.pi, np.pi, (h, w))
    a, b = 100 + 20 * rng.random((h, w)), 50 + 20 * rng.random((h, w))
    return np.stack([a + b * np.cos(phi + d) for d in deltas]).astype(np.float32)


def _phase(frames, deltas):
    """Least squares with the given shifts (float32 as they are passed), plus the first shift, wrapped."""
    d = np.asarray(deltas, np.float32).astype(np.float64)
    a = np.stack([np.ones_like(d), np.cos(d), np.sin(d)], 1)
    x = np.linalg.solve(a.T @ a, np.tensordot(a.T, frames.astype(np.float64), 1).reshape(3, -1))
    p = np.arctan2(-x[2], x[1]) + d[0]
    return np.arctan2(np.sin(p), np.cos(p)).reshape(frames.shape[1:])


@pytest.mark.parametrize("first", [0.0, 3.0, -3.1, 7.0, 10.0, -25.0, 1000.0])
def test_phase_for_given_shifts_is_wrapped(glsu, first):
    """Bar 1e-4 rad: the right-hand sides are FP32 sums of four intensities up to
    190 (2^-24 each), over a modulation of at least 50 and a system whose condition
    number is about 2."""
    deltas = first + np.array([0.0, 1.4, 3.0, 4.5])
    f = _frames(4, 37, 65, deltas)
    a = glsu.AIA(4, 65, 37)
    phi, _, _, it, _ = a.run(list(f), deltas, max_iter=0)
    a.close()
    ref = _phase(f, deltas)
    assert it == 0
    assert phi.min() >= -np.pi - 1e-6 and phi.max() <= np.pi + 1e-6
    assert np.abs(np.angle(np.exp(1j * (phi - ref)))).max() <= 1e-4


def _xy(column, deltas):
    """The two cofactor sums of one pixel in 64 bits, as IEEE arithmetic gives them (right-hand sides in FP32)."""
    d = np.asarray(deltas, np.float32).astype(np.float64)
    c, s = np.cos(d), np.sin(d)
    a = np.stack([np.ones_like(d), c, s], 1)
    cof = np.linalg.inv(a.T @ a) * np.linalg.det(a.T @ a)
    b = [np.float32(0)] * 3
    for v, ck, sk in zip(column, c.astype(np.float32), s.astype(np.float32)):
        b = [np.float32(b[0] + v), np.float32(b[1] + v * ck), np.float32(b[2] + v * sk)]
    return [cof[r, 0] * np.float64(b[0]) + cof[r, 1] * np.float64(b[1]) + cof[r, 2] * np.float64(b[2]) for r in (1, 2)]


@pytest.mark.parametrize("frame", [0, 1, 2, 3])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_pixels_that_are_not_finite(glsu, bad, frame):
    """Without an iteration such a pixel's phase is what 64-bit arithmetic makes of
    it (mostly NaN), the others' what it is without it.  With iterations a run ends as
    not positive definite where the pixel's unit vector is infinity over infinity."""
    deltas = np.array([0.3, 1.7, 3.3, 4.8])
    f = _frames(4, 37, 65, deltas)
    a = glsu.AIA(4, 65, 37)
    good, _, _, _, _ = a.run(list(f), deltas, max_iter=0)
    f[frame, 5, 7] = bad
    phi, _, _, _, _ = a.run(list(f), deltas, max_iter=0)
    with np.errstate(invalid="ignore"):
        x, y = _xy(f[:, 5, 7], deltas)
        want = np.angle(np.exp(1j * (np.arctan2(-y, x) + np.float64(np.float32(deltas[0])))))
        infinite = np.isinf(np.hypot(x, y))
    assert np.isnan(phi[5, 7]) if np.isnan(want) else abs(np.angle(np.exp(1j * (phi[5, 7] - want)))) <= 1e-4
    phi[5, 7] = good[5, 7]
    assert np.array_equal(phi, good)
    if infinite:
        with pytest.raises(glsu.GlsuError) as e:
            a.run(list(f), deltas, max_iter=5)
        assert e.value.code == glsu.ERR_NOT_POSDEF
    a.close()


def test_frames_near_the_range_of_fp32(glsu):
    """Intensities whose products with the system's cofactors pass FP32's range give
    the phases of the same frames scaled down (bar of the given shifts' phases)."""
    deltas = np.array([0.3, 1.7, 3.3, 4.8])
    f = _frames(4, 37, 65, deltas)
    a = glsu.AIA(4, 65, 37)
    small, _, _, _, _ = a.run(list(f), deltas, max_iter=0)
    large, _, _, _, _ = a.run(list(np.ldexp(f, 118)), deltas, max_iter=0)
    a.close()
    assert np.abs(np.angle(np.exp(1j * (small.astype(np.float64) - large)))).max() <= 1e-4
