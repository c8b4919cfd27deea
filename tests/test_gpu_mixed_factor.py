"""The mixed path's FP32 factorisation (128-column blocks, one launch) against
the plain path on active sets below, at and past one, two and three blocks.

Tolerance: -2 log(evidence) within the mixed path's stated 0.2; log det F and
log det R to first order within M 2^-22 k of an FP32 factor whose products
carry 22 bits, k = 1e3 bounding these matrices' condition at lambda = 5 (2e3
at most, and the error is a random sum of M terms)."""
import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu

SIDES = [(3, 3), (11, 11), (12, 11), (12, 12), (17, 16), (20, 20), (23, 22)]


def test_log_dets_match_the_plain_path():
    from qlens_gb300 import PixelLikelihood, abi
    g = Golden("tiny_sie")
    out = []
    for precision in (abi.QLP_FP64, abi.QLP_MIXED):
        pl = PixelLikelihood.from_opts(g.image, g.psf, g.opts, precision=precision)
        pl.set_lens_model(g.lenses, *g.zbeta())
        pl.set_batch_slots(3)
        P = np.tile(np.array(g.params()), (len(SIDES), 1))
        out.append(pl.eval_batch(P, src_sizes=SIDES))
        pl.close()
    for a, b, size in zip(*out, SIDES):
        assert a["status"] == b["status"] == 0
        M = a["n_active_src"]
        assert b["n_active_src"] == M and b["L_nnz"] == a["L_nnz"]
        assert abs(a["m2logev"] - b["m2logev"]) < 0.2, size
        for k in ("logdet_F", "logdet_R"):
            assert abs(a[k] - b[k]) <= M * 2.0 ** -22 * 1e3, (size, k, a[k], b[k])
