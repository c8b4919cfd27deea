"""The plain path's L' (PSF convolution by image tiles in fixed point) against the
same sums in extended precision, from the pre-PSF L that the library returns, on an
image whose sides are no multiple of a tile (32 x 8 pixels), for PSFs of one tap,
narrower and wider than a tile, larger than the image, and past what the bordered
taps in shared memory take (31 x 401).

Tolerance, from the grids: with t = min(30 - exponent of the largest tap, 33 - exponent
of their sum), n entries in a cell's column, the taps to 2^-51 of the largest, L to 2^-58 and
the low halves' product below 2^-(t + 29) an entry:
|error| <= 2^-51 max |tap| sum |L| + 2^-58 sum |tap| + n 2^-(t + 29) + 2^-53 |L'|;
where the sums are in FP64, (n + 1) 2^-53 sum |tap L| + 2^-58 sum |tap|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernel(psf):
    # a border of zeros past 33 taps along a side
    core = tuple(min(p, 33) for p in psf)
    a, b = np.meshgrid(np.arange(core[0]) - core[0] // 2, np.arange(core[1]) - core[1] // 2, indexing="ij")
    k = np.exp(-(a * a + b * b) / 8.0) * np.random.default_rng(6).uniform(-0.2, 1.2, core)
    out = np.zeros(psf)
    i, j = psf[0] // 2 - core[0] // 2, psf[1] // 2 - core[1] // 2
    out[i:i + core[0], j:j + core[1]] = 3.0 * k / np.abs(k).sum()
    return out


@pytest.mark.parametrize("psf", [(1, 1), (3, 9), (21, 5), (33, 31), (31, 401)])
def test_sums_match_extended_precision(psf):
    from qlens_gb300 import PixelLikelihood, abi
    nx, ny, pixel, nsplit = 45, 37, 0.06, 2
    rng = np.random.default_rng(5)
    xv = (np.arange(nx + 1) - nx / 2) * pixel
    yv = (np.arange(ny + 1) - ny / 2) * pixel
    X, Y = np.meshgrid((xv[1:] + xv[:-1]) / 2, (yv[1:] + yv[:-1]) / 2, indexing="ij")
    r = np.hypot(X, Y)
    mask = (r < 1.1).astype(np.uint8)
    kernel = _kernel(psf)
    pl = PixelLikelihood(xv, yv, rng.normal(size=(nx, ny)), mask, kernel, covinv=None, bg_noise=0.05, nsplit=nsplit,
                         src_npixels=(15, 17), regparam=5.0, precision=abi.QLP_FP64)
    pl.set_lens_model([{"type": "sple", "params": [0.6, 1.0, 0.0, 0.75, 30.0, 0.02, -0.01]}])
    res = pl.invert_image_surface_brightness_map()
    assert res["status"] == 0
    d = pl.dump(int(mask.sum()) * nsplit ** 2, res)
    N, M = res["n_active_pixels"], res["n_active_src"]
    got = pl.dump_Lpsf(N, M)
    pl.close()
    assert N == mask.sum()                               # every masked pixel is mapped: rows run over the mask, y outer
    pix = [(i, j) for j in range(ny) for i in range(nx) if mask[i, j]]
    ld = np.longdouble
    cells = rng.choice(M, 12, replace=False)
    L = np.zeros((nx, ny, len(cells)), ld)
    for k, c in enumerate(cells):
        for row, (i, j) in enumerate(pix):
            e = slice(d["L_rowptr"][row], d["L_rowptr"][row + 1])
            v = np.float64(0)
            for w in d["L_value"][e][d["L_index"][e] == c]:
                v = v + w                                # merged in the library's order, in FP64
            L[i, j, k] = v
    px, py = psf
    ref, mag = np.zeros_like(L), np.zeros_like(L)
    for a in range(px):
        for b in range(py):
            if kernel[a, b] == 0:
                continue
            di, dj = px // 2 - a, py // 2 - b            # the tapped pixel is (i + di, j + dj)
            i0, i1, j0, j1 = max(0, -di), min(nx, nx - di), max(0, -dj), min(ny, ny - dj)
            if i0 < i1 and j0 < j1:
                t = L[i0 + di:i1 + di, j0 + dj:j1 + dj]
                ref[i0:i1, j0:j1] += ld(kernel[a, b]) * t
                mag[i0:i1, j0:j1] += np.abs(ld(kernel[a, b]) * t)
    taps, top = np.abs(kernel).sum(), np.abs(kernel).max()
    t = min(30 - np.frexp(top)[1], 33 - np.frexp(taps)[1])
    n, size = (L != 0).sum((0, 1)), np.abs(L).sum((0, 1))
    for row, (i, j) in enumerate(pix):
        tol = 2.0 ** -51 * top * size + 2.0 ** -58 * taps + n * 2.0 ** -(t + 29) + 2.0 ** -53 * np.abs(ref[i, j])
        if psf == (31, 401):
            tol = (n + 1) * 2.0 ** -53 * mag[i, j] + 2.0 ** -58 * taps
        err = np.abs(got[row, cells] - ref[i, j])
        assert (err <= tol).all(), (psf, row, float(err.max()), float(tol.min()))


@pytest.mark.parametrize("batch", [False, True])
def test_refused_psf_leaves_the_context_usable(batch):
    # 131 x 127 taps: past the plain path's range, within the mixed path's
    from qlens_gb300 import PixelLikelihood, abi
    nx, pixel = 30, 0.08
    xv = (np.arange(nx + 1) - nx / 2) * pixel
    pl = PixelLikelihood(xv, xv, np.ones((nx, nx)), np.ones((nx, nx), np.uint8), _kernel((131, 127)), covinv=None,
                         bg_noise=0.1, nsplit=1, src_npixels=(6, 6), regparam=5.0, precision=abi.QLP_FP64)
    pl.set_lens_model([{"type": "sple", "params": [0.6, 1.0, 0.0, 0.75, 30.0, 0.02, -0.01]}])
    p = np.array([[0.6, 1.0, 0.0, 0.75, 30.0, 0.02, -0.01]] * 2)
    if batch:
        with pytest.raises(Exception):
            pl.eval_batch(p)
    else:
        assert pl.invert_image_surface_brightness_map()["status"] != 0
    pl.set_precision(abi.QLP_MIXED)
    r = pl.eval_batch(p)[0] if batch else pl.invert_image_surface_brightness_map()
    assert r["status"] == 0
    pl.close()
