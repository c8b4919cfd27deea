"""The graph replays' job ring and the kernels that clear an evaluation's
buffers: more vectors than the ring holds on one slot, and grids of very
different shapes after one another on the same slot, bit for bit the results
of the same vectors evaluated one by one."""
import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu

KEYS = ("m2logev", "chisq0", "logdet_F", "logdet_R", "n_active_src", "L_nnz")


def _ctx(g, precision, opts=None):
    from qlens_gb300 import PixelLikelihood
    pl = PixelLikelihood.from_opts(g.image, g.psf, opts if opts is not None else g.opts, precision=precision)
    pl.set_lens_model(g.lenses, *g.zbeta())
    return pl


def test_more_vectors_than_the_ring():
    from qlens_gb300 import abi
    g = Golden("tiny_sie")
    pl = _ctx(g, abi.QLP_MIXED)
    pl.set_batch_slots(1)
    rng = np.random.default_rng(8)
    few = np.tile(np.array(g.params()), (7, 1))
    few[:, 0] *= rng.uniform(0.95, 1.05, 7)
    few[:, 3] = rng.uniform(0.6, 0.95, 7)
    n = 1100                                        # the ring holds 1024
    res = pl.eval_batch(few[np.arange(n) % 7])
    want = [pl.invert_image_surface_brightness_map(p) for p in few]
    for i, r in enumerate(res):
        assert all(r[k] == want[i % 7][k] for k in KEYS), i
    pl.close()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_grids_of_different_shapes_on_one_slot(precision):
    from qlens_gb300 import abi
    g = Golden("tiny_sie")
    sizes = [(20, 4), (4, 20), (11, 12), (6, 5), (16, 16), (2, 9), (12, 11)]
    pl = _ctx(g, precision)
    pl.set_batch_slots(1)
    P = np.tile(np.array(g.params()), (len(sizes), 1))
    res = pl.eval_batch(P, src_sizes=sizes)
    pl.close()
    for r, size in zip(res, sizes):
        o = abi.srcgrid_defaults()
        for name, _t in abi.qlp_srcgrid_opts._fields_:
            setattr(o, name, getattr(g.opts, name))
        o.npixels_x, o.npixels_y = size
        one = _ctx(g, precision, o)
        want = one.invert_image_surface_brightness_map()
        one.close()
        assert r["status"] == want["status"] == 0
        assert all(r[k] == want[k] for k in KEYS), size
