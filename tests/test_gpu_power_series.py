"""The power law's deflection series on the GPU, whose number of terms is decided in
FP32, against the oracle's, over flattenings from nearly round (a few terms) to ones
whose series passes the tabulated 48 terms, and slopes on both sides of isothermal.

A term too few or too many moves a deflection by 1e-8 of itself; the transcendental
functions differ by a few ulp, amplified at most ~1e2 times by the slope's power near
the centre: 1e-12 of the largest coordinate."""
import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [0.05, 0.2, 0.6, 0.95, 0.9999])
@pytest.mark.parametrize("slope", [0.5, 0.97, 1.6])
def test_source_points_match_oracle(q, slope):
    from oracle import oracle as O
    from qlens_gb300 import PixelLikelihood
    g = Golden("powerlaw")
    pl = PixelLikelihood.from_opts(g.image, g.psf, g.opts)
    pl.set_lens_model(g.lenses, *g.zbeta())
    p = np.array(g.params())
    p[1], p[3], p[4] = slope, q, 37.0
    r = pl.invert_image_surface_brightness_map(p)
    O.evaluate(g.image, g.psf, g.opts, g.lenses, lens_params=p)
    got, ref = pl.dump(g.n_sub, r)["srcpt"], O.get("srcpt")
    pl.close()
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
