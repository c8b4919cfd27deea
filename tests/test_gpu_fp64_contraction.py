"""The plain path's FP64 contraction F = L'^T C^-1 L' by digit products, against
the oracle's FP64 sums, at source grids around the edges of its 64- and
128-cell tiles and masks that leave remainders of its 32-pixel stages and
128-pixel reads, with uniform noise and with a noise map (whose square root
enters the operand).

Tolerance: the digits and the left-out products are ~2^-54 of the rows' largest
entries per term, so F's error is below that of an FP64 sum of the same terms
(N 2^-53 of its diagonal, N <= 448: 5e-14); with these regularised F (condition
number under 1e4) -2 log(evidence) moves by less than 1e-9 of itself.
"""
import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu

REL = 1e-9
# (source grid, outer radius of the mask): 2x2 to 23x17 cells, 32 to 448 pixels
SHAPES = [((2, 2), 0.3), ((8, 8), 0.5), ((9, 8), 0.9), ((12, 11), 0.7), ((16, 8), 1.2), ((16, 16), 1.1), ((23, 17), 1.2)]


@pytest.mark.parametrize("noise_map", [False, True])
def test_contraction_matches_oracle(noise_map):
    from oracle import oracle as O
    from qlens_gb300 import PixelLikelihood, abi, synthetic
    g = Golden("tiny_sie")
    covinv = None
    if noise_map:
        rng = np.random.default_rng(3)
        covinv = 1.0 / (0.03 * rng.uniform(0.5, 2.0, (g.nx, g.ny))) ** 2
    xv, yv = g.arr["xvals"], g.arr["yvals"]
    masks = np.stack([synthetic.annulus_mask(xv, yv, 0.0, r).ravel() for _, r in SHAPES])
    img = lambda m: abi.ImageBuffers(xv, yv, g.arr["data"], m, covinv, g.sc["background_pixel_noise"])
    keep = img(g.arr["mask"])
    pl = PixelLikelihood.from_opts(keep, g.psf, g.opts, precision=abi.QLP_FP64)
    pl.set_lens_model(g.lenses, *g.zbeta())
    pl.set_batch_slots(2)
    pl.set_instance_masks(masks)
    n = len(SHAPES)
    P = np.tile(np.array(g.params()), (n, 1))
    res = pl.eval_batch(P, mask_ids=list(range(n)), src_sizes=[s for s, _ in SHAPES])
    for i, (size, _) in enumerate(SHAPES):
        o = abi.srcgrid_defaults()
        for name, _t in abi.qlp_srcgrid_opts._fields_:
            setattr(o, name, getattr(g.opts, name))
        o.npixels_x, o.npixels_y = size
        ro = O.evaluate(img(masks[i]), g.psf, o, g.lenses, lens_params=P[i])
        r = res[i]
        assert r["status"] == ro["status"] == 0, (i, r["status"], ro["status"])
        assert r["n_active_src"] == ro["n_active_src"] and r["n_active_pixels"] == ro["n_active_pixels"]
        for k in ("m2logev", "logdet_F", "chisq0"):
            assert abs(r[k] - ro[k]) <= REL * max(abs(ro[k]), 1.0), (size, k, r[k], ro[k])
    pl.close()
