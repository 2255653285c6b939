"""The FFT column sweep of FP64 handles (AUTO): every compiled transform
length at the tallest image it takes and the shortest one (one row more than the
length below takes), against the FP64 oracle and the direct kernel.  Bars: those
of the FP64 form (phase 1e-10 rad, 1e-11 of the largest output)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [256, 384, 512, 640, 768, 1024, 1280, 1536, 2048, 3072, 4096]
HALF = 15  # sigma 5


def _run(glsu, f, p, direct):
    import torch
    t = torch.from_numpy(f).cuda()
    out = torch.empty_like(t)
    w = glsu.WFF2(f.shape[1], f.shape[0], "f64", p)
    if direct:
        w.set_method(glsu.METHOD_DIRECT)
    length = w.tuning()["fft_length"]
    w.run(t.data_ptr(), out.data_ptr())
    w.close()
    return out.cpu().numpy(), length


@pytest.mark.parametrize("edge", ["longest", "shortest"])
@pytest.mark.parametrize("k", range(len(LENGTHS)))
def test_every_length_matches_oracle_and_direct(glsu, oracle, k, edge):
    h = LENGTHS[k] - 2 * HALF if edge == "longest" else (LENGTHS[k - 1] if k else 200) - 2 * HALF + 1
    rng = np.random.default_rng(k)
    y, x = np.mgrid[0:h, 0:5].astype(np.float64)
    f = np.exp(1j * (0.3 * x - 0.2 * y)) + 0.3 * (rng.standard_normal((h, 5)) + 1j * rng.standard_normal((h, 5)))
    p = glsu.WffParams(2.0, -0.4, 0.4, 0.5, HALF / 3.0, -0.5, 0.5, 0.21, 0.1)
    out, length = _run(glsu, f, p, False)
    assert length == LENGTHS[k]
    ref, _ = oracle.wff2(f, *p.tuple())
    assert np.abs(out - ref).max() <= 1e-11 * np.abs(ref).max()
    direct, _ = _run(glsu, f, p, True)
    assert np.abs(out - direct).max() <= 1e-11 * np.abs(ref).max()


def test_explicit_fft_stays_refused_and_env_keeps_direct(glsu, monkeypatch):
    p = glsu.WffParams(10.0, -1, 1, 0.1, 10.0, -1, 1, 0.1, 0.2)
    w = glsu.WFF2(64, 256, "f64", p)
    assert w.tuning()["fft_length"] == 384
    with pytest.raises(glsu.GlsuError) as e:
        w.set_method(glsu.METHOD_FFT)
    assert e.value.code == glsu.ERR_UNSUPPORTED
    w.close()
    monkeypatch.setenv("GLSU_AUTOTUNE", "0")
    w = glsu.WFF2(64, 256, "f64", p)
    assert w.tuning()["fft_length"] == 0 and w.tuning()["method"] == glsu.METHOD_DIRECT
    w.close()


@pytest.mark.parametrize("bad", [1e9, 1e300 ** 0.1, np.inf, np.nan])
def test_a_pixel_acts_on_its_rows_only(glsu, bad):
    """One large or non-finite pixel acts on the rows that two column filters connect
    with it (40: the direct kernel is compiled for half-size 20), as with the direct
    kernel; elsewhere the field is as without it, and for finite values the whole
    output is the direct kernel's.  Bar 1e-11 of the output there."""
    rng = np.random.default_rng(3)
    h, w = 400, 90
    y, x = np.mgrid[0:h, 0:w].astype(np.float64)
    f = np.exp(1j * (0.3 * x - 0.2 * y)) + 0.3 * (rng.standard_normal((h, w)) + 1j * rng.standard_normal((h, w)))
    p = glsu.WffParams(3.0, -0.4, 0.4, 0.5, HALF / 3.0, -0.5, 0.5, 0.21, 0.1)
    f[200, 40] = 0
    a, length = _run(glsu, f, p, False)
    assert length == 512
    f[200, 40] = bad
    b, _ = _run(glsu, f, p, False)
    d, _ = _run(glsu, f, p, True)
    far = np.r_[0:200 - 40, 200 + 41:h]
    assert np.abs(a - b)[far].max() <= 1e-11 * np.abs(a).max()
    assert np.abs(d - b)[far].max() <= 1e-11 * np.abs(a).max()
    if np.isfinite(bad):
        assert (np.abs(d - b).max(1) <= 1e-11 * np.abs(d).max(1)).all()


def test_columns_of_a_wide_range(glsu):
    """Rows from 1 to 2^-40 of the largest in every column: the direct kernel's output, row by row."""
    y, x = np.mgrid[0:300, 0:70].astype(np.float64)
    f = np.exp2(-y * 40 / 300) * np.exp(1j * (0.2 * x - 0.1 * y))
    p = glsu.WffParams(3.0, -0.4, 0.4, 0.5, HALF / 3.0, -0.5, 0.5, 0.21, 0.0)
    b, length = _run(glsu, f, p, False)
    assert length == 384
    d, _ = _run(glsu, f, p, True)
    assert (np.abs(d - b).max(1) <= 1e-11 * np.abs(d).max(1)).all()
