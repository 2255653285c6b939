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
