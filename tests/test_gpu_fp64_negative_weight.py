"""The plain path with a noise map that holds a few negative C^-1 among its pixels, which the
FP64 sums take as they come: against the oracle.

Tolerance: as for positive ones, 1e-9 of -2 log(evidence) and log det F (condition number of
F under 1e4 here, by numpy)."""
import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu


def test_matches_oracle():
    from oracle import oracle as O
    from qlens_gb300 import PixelLikelihood, abi
    g = Golden("tiny_sie")
    rng = np.random.default_rng(9)
    covinv = 1.0 / (0.03 * rng.uniform(0.5, 2.0, (g.nx, g.ny))) ** 2
    pix = np.argwhere(g.arr["mask"].reshape(g.nx, g.ny))
    for i, j in pix[rng.choice(len(pix), 12, replace=False)]:
        covinv[i, j] *= -0.1
    image = abi.ImageBuffers(g.arr["xvals"], g.arr["yvals"], g.arr["data"], g.arr["mask"], covinv, 0.0)
    ro = O.evaluate(image, g.psf, g.opts, g.lenses)
    pl = PixelLikelihood.from_opts(image, g.psf, g.opts, precision=abi.QLP_FP64)
    pl.set_lens_model(g.lenses, *g.zbeta())
    r = pl.invert_image_surface_brightness_map()
    b = pl.eval_batch(np.array([g.params()] * 2))
    pl.close()
    assert r["status"] == ro["status"] == 0
    for k in ("m2logev", "logdet_F", "chisq0"):
        assert abs(r[k] - ro[k]) <= 1e-9 * abs(ro[k]), (k, r[k], ro[k])
        assert all(x[k] == r[k] for x in b)
