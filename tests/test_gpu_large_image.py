"""The plain path on an image of more tiles than one pass of their bitmap holds (393,216 of
32 x 8 pixels), its mask in the last of them: the same L' and likelihood as of the image
cut to the mask's surroundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_same_as_the_cut_out():
    from qlens_gb300 import PixelLikelihood, abi
    nx, ny, cut, pixel = 3, 3_400_000, 200, 1e-6
    rng = np.random.default_rng(2)
    xv = (np.arange(nx + 1) - nx / 2) * pixel * 50
    yv = np.arange(ny + 1) * pixel - 1.0
    psf = rng.uniform(0.1, 1.0, (3, 5))
    data = rng.normal(size=(nx, cut))
    out = []
    for first in (ny - cut, 0):
        whole = first > 0
        d = np.zeros((nx, ny if whole else cut))
        m = np.zeros(d.shape, np.uint8)
        d[:, -cut:] = data
        m[:, -150:-20] = 1
        pl = PixelLikelihood(xv, yv if whole else yv[-cut - 1:], d, m, psf / psf.sum(), bg_noise=0.2, nsplit=2,
                             src_npixels=(4, 11), regparam=3.0, precision=abi.QLP_FP64)
        pl.set_lens_model([{"type": "sple", "params": [0.3, 1.0, 0.0, 0.8, 20.0, 0.1, -0.2]}])
        r = pl.invert_image_surface_brightness_map()
        assert r["status"] == 0 and r["n_active_pixels"] == 3 * 130
        out.append((r, pl.dump_Lpsf(r["n_active_pixels"], r["n_active_src"])))
        pl.close()
    assert np.array_equal(out[0][1], out[1][1])
    for k in ("m2logev", "chisq0", "logdet_F"):
        assert out[0][0][k] == out[1][0][k]
