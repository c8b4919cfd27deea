"""The plain path's factorisation and solves (64-column blocks, digit products,
pivot blocks in 64-bit integers) against the oracle's FP64 ones: active sets
below, at and past one, two and three 64-cell blocks, lambda down to where the
pivot blocks' inverses leave the integers' first range, and no regularisation.

Tolerance: to first order log det F moves by tr(F^-1 dF) <= M k 2^-53 c for a
backward error of c 2^-53 of F, and s by k 2^-53 c of itself; c = 8 allows for
either side's own rounding.  k bounds the condition number of these F (up to
2e3, 4e7 and 1e10 by numpy on such grids).
"""
import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
SIDES = [(3, 3), (8, 8), (9, 8), (12, 11), (14, 14), (20, 17)]


def _opts(g, size, regularization=1):
    from qlens_gb300 import abi
    o = abi.srcgrid_defaults()
    for name, _t in abi.qlp_srcgrid_opts._fields_:
        setattr(o, name, getattr(g.opts, name))
    o.npixels_x, o.npixels_y = size
    o.regularization = regularization
    return o


@pytest.mark.parametrize("lam,k", [(5.0, 1e4), (1e-3, 1e8), (1e-6, 1e11)])
def test_factor_and_solve_match_oracle(lam, k):
    from oracle import oracle as O
    from qlens_gb300 import PixelLikelihood, abi
    g = Golden("tiny_sie")
    pl = PixelLikelihood.from_opts(g.image, g.psf, g.opts, precision=abi.QLP_FP64)
    pl.set_lens_model(g.lenses, *g.zbeta())
    pl.set_batch_slots(3)
    P = np.tile(np.array(g.params()), (len(SIDES), 1))
    res = pl.eval_batch(P, regparams=[lam] * len(SIDES), src_sizes=SIDES)
    for r, size in zip(res, SIDES):
        ro = O.evaluate(g.image, g.psf, _opts(g, size), g.lenses, lens_params=P[0], regparam=lam)
        assert r["status"] == ro["status"] == 0 and r["n_active_src"] == ro["n_active_src"]
        M = r["n_active_src"]
        for name in ("logdet_F", "logdet_R"):
            kk = k if name == "logdet_F" else 1e6
            assert abs(r[name] - ro[name]) <= 8 * EPS * M * kk + 8 * EPS * abs(ro[name]), (size, name)
        tol = 8 * EPS * k * max(abs(ro["chisq0"]), abs(ro["regterms"])) + 8 * EPS * M * 1e6 + 1e-10
        for name in ("chisq0", "m2logev"):
            assert abs(r[name] - ro[name]) <= tol + 8 * EPS * M * k, (size, name, r[name], ro[name])
    pl.close()


def test_no_regularisation():
    from oracle import oracle as O
    from qlens_gb300 import PixelLikelihood, abi
    g = Golden("tiny_sie")
    o = _opts(g, (8, 8), 0)
    pl = PixelLikelihood.from_opts(g.image, g.psf, o, precision=abi.QLP_FP64)
    pl.set_lens_model(g.lenses, *g.zbeta())
    r = pl.invert_image_surface_brightness_map()
    ro = O.evaluate(g.image, g.psf, o, g.lenses)
    assert r["status"] == ro["status"] == 0
    # F alone: condition number under 1e6 (448 pixels on 64 cells)
    assert abs(r["chisq0"] - ro["chisq0"]) <= 8 * EPS * 1e6 * abs(ro["chisq0"])
    assert abs(r["m2logev"] - ro["m2logev"]) <= 8 * EPS * 1e6 * abs(ro["m2logev"])
    pl.close()
