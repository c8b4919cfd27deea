"""The batch's launch schedules -- one, two to eight, and more evaluations in flight take
factorisation grids and graphs of their own -- give the same bits, on both paths, for source
grids of one to several blocks of columns."""
import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu

SIDES = [(8, 8), (12, 11), (20, 17), (26, 26), (16, 16), (30, 24), (9, 8), (22, 20), (13, 12), (28, 30)]


@pytest.mark.parametrize("regopt", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_same_bits_whatever_is_in_flight(precision, regopt):
    from qlens_gb300 import PixelLikelihood
    g = Golden("cfg1")
    pl = PixelLikelihood.from_opts(g.image, g.psf, g.opts, precision=precision)
    pl.set_lens_model(g.lenses, *g.zbeta())
    if regopt:
        pl.set_regparam_optimization(True)
    P = np.tile(np.array(g.params()), (len(SIDES), 1))
    P[:, 0] *= 1.0 + 1e-3 * np.arange(len(SIDES))
    ref = None
    for slots in (1, 2, 8, 9, 10, 3):
        pl.set_batch_slots(slots)
        out = pl.eval_batch(P, src_sizes=SIDES)
        assert all(r["status"] == 0 for r in out)
        if ref is None:
            ref = out
        for a, b in zip(ref, out):
            for k in ("m2logev", "chisq0", "logdet_F", "logdet_R", "Es_times_two", "regparam"):
                assert a[k] == b[k], (slots, k, a[k], b[k])
    pl.close()
