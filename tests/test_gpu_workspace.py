"""R's factor in a band's storage that turns round: log det R on long source grids (two to
thirteen blocks of columns, a few of them within the band) against the oracle, and what a
slot's workspace takes at 4,096 cells.

Tolerance of log det R: M 8 2^-53 k (FP64) and M 2^-22 1e3 (mixed: an FP32 factor whose
products carry 22 bits), k = 1e5 above the condition numbers of these curvature matrices
(4e4 at most, by numpy).
"""
import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu

SIDES = [(4, 200), (3, 90), (60, 5), (24, 33)]


def _opts(g, size):
    from qlens_gb300 import abi
    o = abi.srcgrid_defaults()
    for name, _t in abi.qlp_srcgrid_opts._fields_:
        setattr(o, name, getattr(g.opts, name))
    o.npixels_x, o.npixels_y = size
    return o


@pytest.mark.parametrize("precision", [0, 1])
def test_logdet_R_of_long_grids(precision):
    from oracle import oracle as O
    from qlens_gb300 import PixelLikelihood
    g = Golden("cfg1")
    pl = PixelLikelihood.from_opts(g.image, g.psf, g.opts, precision=precision)
    pl.set_lens_model(g.lenses, *g.zbeta())
    P = np.array(g.params())
    pl.set_batch_slots(2)
    batch = pl.eval_batch(np.tile(P, (len(SIDES), 1)), src_sizes=SIDES)
    pl.close()
    for size, b in zip(SIDES, batch):
        o = _opts(g, size)
        ro = O.evaluate(g.image, g.psf, o, g.lenses, lens_params=P)
        one = PixelLikelihood.from_opts(g.image, g.psf, o, precision=precision)
        one.set_lens_model(g.lenses, *g.zbeta())
        r = one.invert_image_surface_brightness_map()
        one.close()
        M = ro["n_active_src"]
        assert M == r["n_active_src"] == b["n_active_src"] and r["status"] == b["status"] == 0
        tol = M * (8 * 2.0 ** -53 * 1e5 if precision == 0 else 2.0 ** -22 * 1e3)
        assert abs(r["logdet_R"] - ro["logdet_R"]) <= tol, (size, r["logdet_R"], ro["logdet_R"], tol)
        assert b["logdet_R"] == r["logdet_R"]


@pytest.mark.parametrize("precision,per_cell2", [(0, 41), (1, 13)])
def test_slot_memory(precision, per_cell2):
    """Bytes a cell squared at 4,096 cells and few pixels: FP64 F and R 8 each, the digits of
    F's factor 16, the contraction's integers 8.25; mixed F and R 4 each, F's split factor 4."""
    torch = pytest.importorskip("torch")
    from qlens_gb300 import PixelLikelihood
    g = Golden("tiny_sie")
    free0 = torch.cuda.mem_get_info()[0]
    pl = PixelLikelihood.from_opts(g.image, g.psf, _opts(g, (64, 64)), precision=precision)
    pl.set_lens_model(g.lenses, *g.zbeta())
    assert pl.invert_image_surface_brightness_map()["status"] == 0
    used = free0 - torch.cuda.mem_get_info()[0]
    pl.close()
    assert used <= per_cell2 * 4096 ** 2 + (64 << 20), used
