"""The lambda optimisation where no trial has a finite objective (a NaN in the data): the
result is that evaluation's, not one left over from an earlier call."""
import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_result_is_of_this_evaluation(precision):
    from qlens_gb300 import PixelLikelihood, abi
    g = Golden("tiny_sie")
    mask = g.arr["mask"].reshape(g.nx, g.ny)
    i, j = np.argwhere(mask)[len(np.argwhere(mask)) // 2]
    data = np.array(g.arr["data"], float).reshape(g.nx, g.ny).copy()
    data[i, j] = np.nan
    without = mask.copy()
    without[i, j] = 0
    image = abi.ImageBuffers(g.arr["xvals"], g.arr["yvals"], data, mask, None, g.sc["background_pixel_noise"])
    pl = PixelLikelihood.from_opts(image, g.psf, g.opts, precision=precision)
    pl.set_lens_model(g.lenses, *g.zbeta())
    pl.set_instance_masks(without.reshape(1, -1))
    pl.set_regparam_optimization(True)
    P = np.array([g.params()])
    good = pl.eval_batch(P, mask_ids=[0])[0]
    assert good["status"] == 0 and np.isfinite(good["chisq0"])
    bad = pl.eval_batch(P, mask_ids=[-1])[0]
    pl.close()
    assert bad["n_active_pixels"] == good["n_active_pixels"] + 1
    assert np.isnan(bad["chisq0"]) and np.isnan(bad["m2logev"])
