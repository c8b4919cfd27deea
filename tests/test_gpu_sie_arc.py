"""The core-free isothermal lens in the FP64 pre-pass of the surrogate's ray shooting (polynomials
of its two arc functions) against the oracle: a halo of no mass on the same plane sends the rays
that way and adds nothing.  Axis ratios from round (arguments below the table's 2^-20)
over its range to thinner than 1/64 (past its 2^12).

Tolerance: a few roundings, and the oracle's own atanh(z), whose derivative 1 / (1 - z^2) is at most
1 / q^2: (1e-14 + 2e-15 / q^2) of the largest coordinate and the lens strength."""
import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def trained():
    from qlens_gb300 import pixlike
    return pixlike.train_nfw_surrogate(steps=64, n_train=1 << 16, batch=4096)


@pytest.mark.parametrize("q", [0.012, 0.05, 0.3, 0.75, 0.9999, 0.99999999])
@pytest.mark.parametrize("theta", [0.0, 33.0])
def test_source_points_match_oracle(trained, q, theta):
    from oracle import oracle as O
    from qlens_gb300 import PixelLikelihood, abi
    g = Golden("nfw")
    pl = PixelLikelihood.from_opts(g.image, g.psf, g.opts, precision=abi.QLP_MIXED)
    pl.set_lens_model(g.lenses, *g.zbeta())
    pl.set_nfw_mode(abi.QLP_NFW_SURROGATE)
    p = np.array(g.params())
    p[1], p[2], p[3], p[4] = 1.0, 0.0, q, theta
    p[11] = 1e-40                                        # the halo's ks
    r = pl.invert_image_surface_brightness_map(p)
    O.evaluate(g.image, g.psf, g.opts, g.lenses, lens_params=p, planes=g.planes())
    got, ref = pl.dump(g.n_sub, r)["srcpt"], O.get("srcpt")
    pl.close()
    assert np.abs(got - ref).max() <= (1e-14 + 2e-15 / q ** 2) * (np.abs(ref).max() + p[0])


@pytest.mark.parametrize("n", [3, 17, 66, 131])
def test_ray_groups(trained, n):
    # 81 rays (less than a group of 128) to 1,206 groups (3.97 for each of 304 in flight)
    from qlens_gb300 import PixelLikelihood, abi
    xv = (np.arange(n + 1) - n / 2) * (4.0 / n)
    sie = [{"type": "sple", "params": [1.1, 1.0, 0.0, 0.7, 20.0, 0.01, -0.02]}]
    halo = [{"type": "nfw", "params": [1e-40, 2.0, 0.8, 10.0, 0.3, 0.2]}]
    got = []
    for lenses, precision in ((sie, abi.QLP_FP64), (sie + halo, abi.QLP_MIXED)):
        pl = PixelLikelihood(xv, xv, np.ones((n, n)), np.ones((n, n), np.uint8), np.ones((1, 1)), covinv=None,
                             bg_noise=0.1, nsplit=3, src_npixels=(8, 8), regparam=5.0, precision=precision)
        pl.set_lens_model(lenses)
        if precision == abi.QLP_MIXED:
            pl.set_nfw_mode(abi.QLP_NFW_SURROGATE)
        r = pl.invert_image_surface_brightness_map()
        got.append(pl.dump(9 * n * n, r)["srcpt"])
        pl.close()
    assert np.abs(got[1] - got[0]).max() <= 2e-14 * (np.abs(got[0]).max() + 1.1)
