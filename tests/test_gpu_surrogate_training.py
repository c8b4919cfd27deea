"""The training step's kernels at the edges of their row tiles: batches of one
row, of a ragged split, and on either side of each tile height (2, 4, 7 and 8
rows a thread), loss and gradients against the CPU oracle with the bounds of the
512-row check."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [3, 128, 128, 128, 128, 2]


@pytest.mark.parametrize("rows", [1, 31, 511, 4864, 4865, 9729, 17024, 17025, 19457])
def test_gradients_match_oracle(rows):
    from oracle import oracle as O
    from qlens_gb300 import pixlike
    rng = np.random.default_rng(rows)
    p = np.concatenate([v for a, b in zip(DIMS[:-1], DIMS[1:])
                        for v in (rng.uniform(-1, 1, a * b) * np.sqrt(6.0 / (a + b)), rng.normal(0, 0.05, b))])
    p = p.astype(np.float32)
    x = rng.uniform(-1, 1, (rows, 3)).astype(np.float32)
    t = rng.normal(0, 1, (rows, 2)).astype(np.float32)
    loss, grad = pixlike.surrogate_grad_check(p, x, t)
    loss_o, grad_o, _ = O.mlp_loss_grad(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64))
    assert abs(loss - loss_o) <= 1e-4 * abs(loss_o)
    o = 0
    for a, b in zip(DIMS[:-1], DIMS[1:]):
        for n in (a * b, b):
            g, go = grad[o:o + n].astype(np.float64), grad_o[o:o + n]
            assert np.linalg.norm(g - go) < 2e-3 * max(np.linalg.norm(go), 1e-30), (a, b, n)
            o += n
