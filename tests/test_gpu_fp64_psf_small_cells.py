"""The plain path's L' of source cells that only the edge of one sub-pixel's footprint
touches (weights of 1e-3 to 1e-12, the whole column of L): as accurate relative to the cell's own
largest L' as any other cell's.  The source grid is laid so that the sub-pixel with the
largest x lies that fraction of a cell past a cell's centre.

Tolerance, relative to sum |tap| max |L| of the cell: taps to 2^-51 of the largest and L to
2^-58 of the cell's largest, a term each; the low halves' product and the final rounding
below 2^-51.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENS = [{"type": "sple", "params": [0.6, 1.0, 0.0, 0.75, 30.0, 0.02, -0.01]}]
NX, CELLS = 24, (8, 9)


def _context(grid):
    from qlens_gb300 import PixelLikelihood, abi
    rng = np.random.default_rng(4)
    xv = (np.arange(NX + 1) - NX / 2) * 0.08
    a = np.exp(-np.add.outer(np.arange(-2, 3) ** 2, np.arange(-2, 3) ** 2) / 3.0)
    pl = PixelLikelihood(xv, xv, rng.normal(size=(NX, NX)), np.ones((NX, NX), np.uint8), a / a.sum(), bg_noise=0.05, nsplit=2,
                         src_npixels=CELLS, auto_sourcegrid=False, sourcegrid=grid, regparam=5.0, precision=abi.QLP_FP64)
    pl.set_lens_model(LENS)
    res = pl.invert_image_surface_brightness_map()
    assert res["status"] == 0
    return pl, res, pl.dump(4 * NX * NX, res), a / a.sum()


@pytest.mark.parametrize("weight", [1e-3, 1e-6, 1e-9, 1e-12])
def test_relative_to_the_cells_own_largest(weight):
    pl, _res, d, _psf = _context((-3.0, 3.0, -3.0, 3.0))
    pl.close()
    x = d["srcpt"][0::2].max()
    y = np.abs(d["srcpt"][1::2]).max()
    # the centre of column 5 of 8 lies weight cells left of x
    step = 0.25
    left = x - weight * step - 5.5 * step
    pl, res, d, psf = _context((left, left + CELLS[0] * step, -1.2 * y, 1.2 * y))
    N, M = res["n_active_pixels"], res["n_active_src"]
    got = pl.dump_Lpsf(N, M)
    pl.close()
    L = np.zeros((N, M), np.longdouble)
    for row in range(N):
        for e in range(d["L_rowptr"][row], d["L_rowptr"][row + 1]):
            L[row, d["L_index"][e]] = np.float64(L[row, d["L_index"][e]]) + d["L_value"][e]
    small = [c for c in range(M) if 0 < np.abs(L[:, c]).max() < 2 * weight]
    assert small, "no cell is touched by the edge alone"
    assert N == NX * NX                                # every pixel is mapped: rows run over the image, y outer
    h = psf.shape[0] // 2
    for c in small:
        img = L[:, c].reshape(NX, NX).T                # [i, j]
        ref = np.zeros_like(img)
        for a in range(5):
            for b in range(5):
                di, dj = h - a, h - b
                i0, i1, j0, j1 = max(0, -di), min(NX, NX - di), max(0, -dj), min(NX, NX - dj)
                ref[i0:i1, j0:j1] += np.longdouble(psf[a, b]) * img[i0 + di:i1 + di, j0 + dj:j1 + dj]
        n = int((img != 0).sum())
        tol = (n * (2.0 ** -51 + 2.0 ** -58) + 2.0 ** -51) * float(np.abs(img).max()) * np.abs(psf).sum()
        err = np.abs(got[:, c] - ref.T.reshape(-1))
        assert (err <= tol).all(), (weight, c, float(err.max()), tol)
