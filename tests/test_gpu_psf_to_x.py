"""The mixed path's PSF-to-X build against the plain path, on an image whose
sides are no multiple of a tile (32 x 8 pixels), for PSFs of one tap, narrower and
wider than a tile and larger than the image, with few and many entries a column.
Past what the bordered taps in shared memory take (131 x 127; the plain path does
not take that many) the same PSF in a border of zeros gives F's same bits (the
right-hand side's convolutions have kernels of their own for such a PSF).

X enters F alone: log det F to first order within M 2^-22 k of the products'
22 bits, k = 1e3 bounding these matrices' condition at lambda = 5, and
-2 log(evidence) within the mixed path's stated 0.2; X's sparsity is the plain
path's (n_active_src, L_nnz equal)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("m2logev", "chisq0", "logdet_F", "logdet_R", "Es_times_two", "regterms", "n_active_src", "L_nnz",
        "n_active_pixels")


def _evaluate(kernel, src, precision):
    from qlens_gb300 import PixelLikelihood
    nx, ny, pixel = 45, 37, 0.06
    rng = np.random.default_rng(5)
    xv = (np.arange(nx + 1) - nx / 2) * pixel
    yv = (np.arange(ny + 1) - ny / 2) * pixel
    X, Y = np.meshgrid((xv[1:] + xv[:-1]) / 2, (yv[1:] + yv[:-1]) / 2, indexing="ij")
    r = np.hypot(X, Y)
    data = np.exp(-((r - 0.6) / 0.15) ** 2) + 0.05 * rng.normal(size=(nx, ny))
    mask = (r < 1.1).astype(np.uint8)
    pl = PixelLikelihood(xv, yv, data, mask, kernel, covinv=None, bg_noise=0.05, nsplit=2, src_npixels=src,
                         regparam=5.0, precision=precision)
    pl.set_lens_model([{"type": "sple", "params": [0.6, 1.0, 0.0, 0.75, 30.0, 0.02, -0.01]}])
    out = [pl.invert_image_surface_brightness_map() for _ in range(2)]
    pl.close()
    assert out[0]["status"] == 0
    assert all(out[0][k] == out[1][k] for k in KEYS)      # X was left all zero
    return out[0]


def _kernel(psf):
    a, b = np.meshgrid(np.arange(psf[0]) - psf[0] // 2, np.arange(psf[1]) - psf[1] // 2, indexing="ij")
    kernel = np.exp(-(a * a + b * b) / 8.0) * np.random.default_rng(6).uniform(0.8, 1.2, psf)
    return kernel / kernel.sum()


@pytest.mark.parametrize("psf", [(1, 1), (3, 9), (21, 5), (33, 31), (61, 45)])
@pytest.mark.parametrize("src", [(4, 3), (15, 17)])
def test_log_det_matches_the_plain_path(psf, src):
    from qlens_gb300 import abi
    p, m = (_evaluate(_kernel(psf), src, precision) for precision in (abi.QLP_FP64, abi.QLP_MIXED))
    for k in ("n_active_src", "L_nnz", "n_active_pixels"):
        assert p[k] == m[k]
    assert abs(p["m2logev"] - m["m2logev"]) < 0.2
    assert abs(p["logdet_F"] - m["logdet_F"]) <= p["n_active_src"] * 2.0 ** -22 * 1e3


def test_taps_past_shared_memory():
    from qlens_gb300 import abi
    kernel = _kernel((61, 45))
    wide = np.zeros((131, 127))
    wide[35:96, 41:86] = kernel
    a, b = (_evaluate(k, (15, 17), abi.QLP_MIXED) for k in (kernel, wide))
    assert a["logdet_F"] == b["logdet_F"] and a["L_nnz"] == b["L_nnz"]


def test_more_pixels_than_the_contraction_lists_at_once():
    # 4,096 stages of 64 pixels a stretch: 262,144 pixels, and a second stretch past them
    from qlens_gb300 import PixelLikelihood, abi
    n, pixel = 530, 0.004
    rng = np.random.default_rng(9)
    xv = (np.arange(n + 1) - n / 2) * pixel
    data = 0.05 * rng.normal(size=(n, n))
    out = []
    for precision in (abi.QLP_FP64, abi.QLP_MIXED):
        pl = PixelLikelihood(xv, xv, data, np.ones((n, n), np.uint8), _kernel((3, 3)), covinv=None, bg_noise=0.05,
                             nsplit=1, src_npixels=(9, 16), regparam=5.0, precision=precision)
        pl.set_lens_model([{"type": "sple", "params": [0.6, 1.0, 0.0, 0.75, 30.0, 0.02, -0.01]}])
        out.append(pl.invert_image_surface_brightness_map())
        pl.close()
    p, m = out
    assert p["n_active_pixels"] > 4096 * 64 and all(p[k] == m[k] for k in ("n_active_src", "L_nnz", "n_active_pixels"))
    assert abs(p["logdet_F"] - m["logdet_F"]) <= p["n_active_src"] * 2.0 ** -22 * 1e3
