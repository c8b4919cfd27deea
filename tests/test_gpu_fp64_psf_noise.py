"""The plain path's L' under a noise map: entries that are small for their taps can carry
the largest weights sqrt(C^-1), so L' is then as accurate for each entry as an FP64 sum of
it, not for the cell's largest one only.  A PSF with a core of 1 and wings of 1e-7, noise maps
whose sqrt(C^-1) spans 1e8 in the image's mask or in a batch's, against extended precision.

Tolerance: an FP64 sum of n terms, (n + 1) 2^-53 sum |tap L|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX = 28


def _problem():
    rng = np.random.default_rng(8)
    xv = (np.arange(NX + 1) - NX / 2) * 0.08
    X, Y = np.meshgrid((xv[1:] + xv[:-1]) / 2, (xv[1:] + xv[:-1]) / 2, indexing="ij")
    mask = (np.hypot(X, Y) < 0.9).astype(np.uint8)
    kernel = 1e-7 * rng.uniform(0.3, 1.0, (7, 7))
    kernel[3, 3] = 1.0
    return xv, rng.normal(size=(NX, NX)), mask, kernel


def _check(pl, res, mask, kernel, nsplit):
    d = pl.dump(int(mask.sum()) * nsplit ** 2, res)
    N, M = res["n_active_pixels"], res["n_active_src"]
    got = pl.dump_Lpsf(N, M)
    assert N == mask.sum()
    pix = [(i, j) for j in range(NX) for i in range(NX) if mask[i, j]]
    L = np.zeros((NX, NX, M), np.longdouble)
    for row, (i, j) in enumerate(pix):
        for e in range(d["L_rowptr"][row], d["L_rowptr"][row + 1]):
            L[i, j, d["L_index"][e]] = np.float64(L[i, j, d["L_index"][e]]) + d["L_value"][e]
    ref, mag, n = np.zeros_like(L), np.zeros_like(L), np.zeros(L.shape, int)
    h = kernel.shape[0] // 2
    for a in range(kernel.shape[0]):
        for b in range(kernel.shape[1]):
            di, dj = h - a, h - b
            i0, i1, j0, j1 = max(0, -di), min(NX, NX - di), max(0, -dj), min(NX, NX - dj)
            t = np.longdouble(kernel[a, b]) * L[i0 + di:i1 + di, j0 + dj:j1 + dj]
            ref[i0:i1, j0:j1] += t
            mag[i0:i1, j0:j1] += np.abs(t)
            n[i0:i1, j0:j1] += t != 0
    for row, (i, j) in enumerate(pix):
        err = np.abs(got[row] - ref[i, j])
        tol = (n[i, j] + 1) * 2.0 ** -53 * mag[i, j]
        assert (err <= tol).all(), (row, float((err / np.maximum(tol, 1e-300)).max()))


@pytest.mark.parametrize("where", ["mask", "batch"])
def test_entries_as_accurate_as_fp64_sums(where):
    from qlens_gb300 import PixelLikelihood, abi
    xv, data, mask, kernel = _problem()
    s = 3.0 * np.where(np.arange(NX)[:, None] % 2 == 0, 1.0, 1e8) + np.zeros((NX, NX))
    if where == "batch":                     # the extremes lie in another mask only
        s = np.where(mask == 1, 3.0, s)
    other = np.ones((NX, NX), np.uint8)
    pl = PixelLikelihood(xv, xv, data, mask, kernel, covinv=s * s, nsplit=2, src_npixels=(9, 10), regparam=5.0,
                         precision=abi.QLP_FP64)
    pl.set_lens_model([{"type": "sple", "params": [0.6, 1.0, 0.0, 0.75, 30.0, 0.02, -0.01]}])
    if where == "batch":
        pl.set_instance_masks(other.reshape(1, -1))
        # an evaluation on the extended set of pixels; the image's own mask is then summed alike
        b = pl.eval_batch(np.array([[0.6, 1.0, 0.0, 0.75, 30.0, 0.02, -0.01]] * 2), mask_ids=[0, 0])
        assert all(r["n_active_pixels"] > mask.sum() for r in b)
    res = pl.invert_image_surface_brightness_map()
    assert res["status"] in (0, abi.QLP_ERR_NOT_SPD)
    _check(pl, res, mask, kernel, 2)
    pl.close()
