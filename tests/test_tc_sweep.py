"""The tensor-core column sweep of the FP32 WFF2 (GLSU_METHOD_FFT without an
FFT plan set by hand) at the sizes where its tiling can go wrong: one row and
one column, the 16-row steps, the tile heights (64, 128, 160 rows), the 64
columns of a tile, odd heights (rows are kept in pairs), the half-sizes at which
the MMA width N = roundup16(2s + 16) and the tile height change, and the
largest half-size it takes.

Tolerance against the FP64 oracle, with threshold 0 so that no pixel can
flip: per pass at most 24 truncated accumulations (2^-23 each) and the
operands' split (2^-22), two passes, and two FP32 row filters of up to 97
taps (2^-24 a term at worst, twice): below 2e-5 of the largest output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-5


def _field(shape, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:shape[0], 0:shape[1]].astype(np.float64)
    f = np.exp(1j * (0.3 * x - 0.2 * y + 0.002 * x * y)) * (1 + 0.5 * np.cos(x / 9.0))
    return (f + 0.2 * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))).astype(np.complex64)


def _run(glsu, f, sigy, n=3, sigx=2.0, thr=0.0, length=None):
    import torch
    p = glsu.WffParams(sigx, -0.4, 0.4, 0.8 / (n - 0.5), sigy, -0.4, 0.4, 0.8 / (n - 0.5), thr)
    t = torch.from_numpy(np.ascontiguousarray(f)).cuda()
    out = torch.full_like(t, float("nan"))
    w = glsu.WFF2(f.shape[1], f.shape[0], "f32", p)
    w.set_method(glsu.METHOD_FFT)
    if length:
        w.set_fft_length(w.tuning()["fft_length"])
    w.run(t.data_ptr(), out.data_ptr())
    w.close()
    return out.cpu().numpy(), p


SHAPES = [(1, 1), (2, 3), (15, 64), (16, 65), (17, 63), (63, 10), (64, 40), (65, 129), (159, 70), (160, 12),
          (161, 33), (321, 66), (500, 20)]


@pytest.mark.parametrize("shape", SHAPES)
def test_tile_edges_match_oracle(glsu, oracle, shape):
    f = _field(shape, 1)
    for sigy in (2.0, 10.0, 16.0):
        out, p = _run(glsu, f, sigy)
        ref, _ = oracle.wff2(f.astype(np.complex128), *p.tuple())
        assert np.abs(out - ref).max() <= TOL * np.abs(ref).max(), (shape, sigy)


@pytest.mark.parametrize("half", [0, 1, 7, 8, 9, 16, 17, 24, 25, 32, 33, 40, 41, 47, 48, 49])
def test_half_sizes_match_oracle(glsu, oracle, half):
    f = _field((203, 70), 2)
    out, p = _run(glsu, f, max(half, 0.1) / 3.0)
    ref, _ = oracle.wff2(f.astype(np.complex128), *p.tuple())
    assert np.abs(out - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("e", [-60, -20, 20, 60])
def test_scaled_input_gives_scaled_bits(glsu, e):
    """The operands' range follows the input's, by powers of two."""
    f = _field((90, 80), 3)
    a, _ = _run(glsu, f, 6.0)
    b, _ = _run(glsu, np.ldexp(f.view(np.float32), e).view(np.complex64), 6.0)
    assert np.array_equal(np.ldexp(a.view(np.float32), e), b.view(np.float32))


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_pixel_stays_in_its_columns(glsu, bad):
    """Columns beyond both row filters' reach of a non-finite pixel are as
    without it.  (The row kernels are compiled for half-sizes 12, 20, ... and
    multiply by zero taps up to that: their reach, here 12, is the compiled one.)"""
    f = _field((120, 200), 4)
    f[50, 30] = 0
    a, _ = _run(glsu, f, 5.0, sigx=4.0)
    f[50, 30] = bad
    b, _ = _run(glsu, f, 5.0, sigx=4.0)
    far = 30 + 2 * 12 + 1
    assert np.array_equal(a[:, far:], b[:, far:])


def test_zero_field_and_high_threshold(glsu):
    f = _field((70, 90), 5)
    for g, thr in ((np.zeros_like(f), 0.0), (f, 1e30)):
        out, _ = _run(glsu, g, 8.0, thr=thr)
        assert np.array_equal(out, np.zeros_like(out))


def test_fft_length_by_hand_runs_the_fft_sweep(glsu):
    """Setting a length selects the FFT kernels, whose bits differ; both agree to the tolerance."""
    f = _field((300, 130), 6)
    a, _ = _run(glsu, f, 10.0, n=5)
    b, _ = _run(glsu, f, 10.0, n=5, length=True)
    assert not np.array_equal(a, b)
    assert np.abs(a - b).max() <= TOL * np.abs(b).max()


@pytest.mark.parametrize("shape,sigma", [((41, 37), 2.0), ((150, 133), 10.0), ((163, 171), 16.0)])
@pytest.mark.parametrize("side", [-1, 1])
def test_threshold_close_to_every_value(glsu, oracle, shape, sigma, side):
    """A plane wave on the grid has |U| = sum(w) for the whole window inside the
    image, and the threshold lies 2e-6 beside it: within the band that is decided in
    FP64, and 10 times what R's and the phasors' FP32 rounding can move |U| by
    (about 2^-24 each, averaged over the window).  All such values pass, or none;
    bar of the FP32 form, 1e-5 of the field."""
    import torch
    h, w = shape
    y, x = np.mgrid[0:h, 0:w].astype(np.float64)
    f = np.exp(1j * (0.25 * x - 0.5 * y)).astype(np.complex64)
    s = int(np.floor(3 * sigma + 0.5))
    n = np.arange(-s, s + 1)
    g = np.exp(-n ** 2 / (2 * sigma ** 2))
    top = g.sum() ** 2 / (g ** 2).sum()
    p = glsu.WffParams(sigma, 0.25, 0.25, 1.0, sigma, -0.5, -0.5, 1.0, top * (1 + side * 2e-6))
    t = torch.from_numpy(f).cuda()
    out = torch.empty_like(t)
    filt = glsu.WFF2(w, h, "f32", p)
    filt.set_method(glsu.METHOD_FFT)
    filt.run(t.data_ptr(), out.data_ptr())
    filt.close()
    ref, _ = oracle.wff2(f.astype(np.complex128), *p.tuple())
    assert (np.abs(ref).max() > 0) == (side < 0)
    assert np.abs(out.cpu().numpy() - ref).max() <= 1e-5 * max(np.abs(ref).max(), 1e-3)


@pytest.mark.parametrize("shape,sigma", [((5, 70), 0.4), ((16, 64), 2.0), ((31, 130), 4.0), ((163, 64), 0.5),
                                         ((161, 200), 1.0)])
def test_one_pair_of_blocks_a_wy(glsu, oracle, shape, sigma):
    """Where a wy has one pair of 16-row blocks (short images, a short last
    tile), the two thresholding warpgroups take it in turns over many wy."""
    f = _field(shape, 7)
    p = glsu.WffParams(2.0, -0.2, 0.2, 0.3, sigma, -1.0, 1.0, 0.01, 0.0)
    import torch
    t = torch.from_numpy(f).cuda()
    w = glsu.WFF2(shape[1], shape[0], "f32", p)
    w.set_method(glsu.METHOD_FFT)
    outs = []
    for _ in range(3):
        out = torch.full_like(t, float("nan"))
        w.run(t.data_ptr(), out.data_ptr())
        outs.append(out.cpu().numpy())
    w.close()
    ref, _ = oracle.wff2(f.astype(np.complex128), *p.tuple())
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])
    assert np.abs(outs[0] - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("size", [1e5, 1e9, 1e30])
def test_a_large_finite_pixel_stays_in_its_columns_and_tiles(glsu, size):
    """Columns beyond both row filters' reach of one large pixel (as for a
    non-finite one), and rows of tiles that do not read it (a tile is at most 160
    rows and reads 2s + 16 more on either side), have the bits they have without
    it.  In the rows of its own tiles and columns that no filter connects with it
    (2s away), R is off by 2^-25 of a value scaled to 2^15: 2^-40 of the pixel."""
    f = _field((700, 200), 8)
    f[50, 30] = 0
    a, _ = _run(glsu, f, 5.0, sigx=4.0)
    f[50, 30] = size
    b, _ = _run(glsu, f, 5.0, sigx=4.0)
    far = 30 + 2 * 12 + 1
    assert np.array_equal(a[:, far:], b[:, far:])
    assert np.array_equal(a[320:], b[320:])
    if size == 1e5:
        top = np.abs(a).max()
        assert np.abs(a - b)[50 + 2 * 15 + 1:].max() <= TOL * top


@pytest.mark.parametrize("bad", [1e9, 1e30, np.inf, np.nan])
def test_auto_keeps_the_direct_kernels_reach(glsu, bad):
    """With a window for which AUTO would take the direct kernel before the FFT
    sweep, one pixel acts on the rows that two column filters connect with it (40, as
    the direct kernel is compiled for half-size 20) and on no others."""
    import torch
    f = _field((500, 200), 10)
    p = glsu.WffParams(4.0, -0.4, 0.4, 0.05, 5.0, -0.4, 0.4, 0.05, 0.0)

    def run(v, direct):
        g = f.copy()
        g[250, 60] = v
        t = torch.from_numpy(g).cuda()
        out = torch.empty_like(t)
        w = glsu.WFF2(200, 500, "f32", p)
        assert w.tuning()["method"] == glsu.METHOD_FFT
        if direct:
            w.set_method(glsu.METHOD_DIRECT)
        w.run(t.data_ptr(), out.data_ptr())
        w.close()
        return out.cpu().numpy()

    a, b, d = run(0, False), run(bad, False), run(bad, True)
    far = np.r_[0:250 - 40, 250 + 41:500]
    assert np.abs(a - b)[far].max() <= TOL * np.abs(a).max()
    assert np.abs(d - b)[far].max() <= TOL * np.abs(a).max()
    if np.isfinite(bad):
        assert np.abs(d - b).max() <= TOL * np.abs(d).max()


def test_wide_columns_over_many_tiles(glsu, oracle):
    """A field whose amplitude falls by 2^20 within every tile, odd sizes: every
    column is done directly; the FP32 form's bar by rows of like size."""
    import torch
    y, x = np.mgrid[0:333, 0:200].astype(np.float64)
    amp = np.exp2(-20.0 * np.abs(((y + 20) % 64) / 32 - 1))
    f = (amp * np.exp(1j * (0.2 * x - 0.1 * y))).astype(np.complex64)
    p = glsu.WffParams(2.0, -0.4, 0.4, 0.05, 2.0, -0.4, 0.4, 0.05, 0.0)
    t = torch.from_numpy(f).cuda()
    out = torch.empty_like(t)
    w = glsu.WFF2(200, 333, "f32", p)
    assert w.tuning()["method"] == glsu.METHOD_FFT
    w.run(t.data_ptr(), out.data_ptr())
    w.close()
    ref, _ = oracle.wff2(f.astype(np.complex128), *p.tuple())
    err = np.abs(out.cpu().numpy() - ref).max(1)
    assert (err <= TOL * np.abs(ref).max(1)).all()


@pytest.mark.parametrize("kind", ["constant", "wave", "noise"])
@pytest.mark.parametrize("half", [15, 30, 45])
def test_error_and_scale_of_a_single_frequency(glsu, oracle, half, kind):
    """The sums' truncation is balanced and its mean taken out.  Uncorrected, the
    output is 2.3, 3.8 and 6.4e-7 too small at these half-sizes (twice a pass's
    loss), and a constant column, whose low parts would all have one sign, is off by
    up to 6e-7 beside that.  Bars of the output's norm: its scale within 2e-7 (0.4e-7
    a pass between kinds of data, and as much for the FP32 row filters), the error
    within 4e-7 (a pass: 3 x 16 products for each of at most 7 steps cut off by up
    to 2^-26, and 21 sums by up to 2^-23, at random: 2.2e-7; twice, and the filters)."""
    import torch
    rng = np.random.default_rng(half)
    H, W = 320, 96
    y = np.arange(H)[:, None]
    amp = np.exp2(rng.uniform(-1, 0, W))[None]
    phase = rng.uniform(0, 2 * np.pi, W)[None]
    if kind == "constant":
        f = amp * np.exp(1j * (phase + 0 * y))
    elif kind == "wave":
        f = amp * np.exp(1j * (phase + 0.02 * y + 2 * np.cos(y / 40.0)))
    else:
        f = rng.standard_normal((H, W)) + 1j * rng.standard_normal((H, W))
    f = f.astype(np.complex64)
    p = glsu.WffParams(0.1, 0.0, 0.0, 1.0, half / 3.0, 0.0, 0.0, 1.0, 0.0)
    t = torch.from_numpy(f).cuda()
    out = torch.empty_like(t)
    w = glsu.WFF2(W, H, "f32", p)
    w.set_method(glsu.METHOD_FFT)
    w.run(t.data_ptr(), out.data_ptr())
    w.close()
    out = out.cpu().numpy().astype(np.complex128)
    ref, _ = oracle.wff2(f.astype(np.complex128), *p.tuple())
    power = (np.abs(ref) ** 2).sum()
    assert abs((np.conj(ref) * (out - ref)).sum().real / power) <= 2e-7
    assert np.sqrt((np.abs(out - ref) ** 2).sum() / power) <= 4e-7
