"""The plain path on matrices F = L'^T C^-1 L' + lambda R that are not positive definite
(lambda < 0): flagged, and log det F and the amplitudes as the reference's Cholesky goes
on, with sqrt(|d|) at a negative pivot, against that factorisation in extended precision of F
summed in extended precision from the oracle's L'; one to three 64-cell blocks.

Tolerance: the factors grow without bound here, so it is taken from the problem: 1e3
times what the same factorisation in FP64 (numpy) is off, and 1e-9 (log det F) or
1e-8 (amplitudes) of the values.  The cases are ones whose log det F moves by less than a
tenth of that when F's entries move by 2^-53 sqrt(F_ii F_jj), an FP64 sum's rounding.
"""
import numpy as np
import pytest

from goldens import Golden
from test_gpu_fp64_noise_range import _curvature

CASES = [((3, 3), -500.0, False), ((8, 8), -0.05, True), ((8, 8), -500.0, False), ((9, 8), -0.01, True),
         ((12, 11), -500.0, False), ((14, 14), -1e-6, False)]


def _factor(F, dtype):
    A = F.astype(dtype)
    negative = False
    for k in range(len(A)):
        negative |= bool(A[k, k] < 0)
        A[k, k] = np.sqrt(abs(A[k, k]))
        A[k + 1:, k] /= A[k, k]
        A[k + 1:, k + 1:] -= np.outer(A[k + 1:, k], A[k + 1:, k])
    return np.tril(A), negative


def _solve(L, D):
    x = D.astype(L.dtype)
    for i in range(len(L)):
        x[i] = (x[i] - L[i, :i] @ x[:i]) / L[i, i]
    for i in range(len(L) - 1, -1, -1):
        x[i] = (x[i] - L[i + 1:, i] @ x[i + 1:]) / L[i, i]
    return x


def _setup(size, lam, patch):
    """(case, image, options, log det F, its tolerance, s, its tolerance, F); patch: the
    pixels of large x nearly without weight."""
    from oracle import oracle as O
    from qlens_gb300 import abi
    g = Golden("tiny_sie")
    c = np.full((g.nx, g.ny), 400.0)
    if patch:
        c[18:, :] = 1e-4
    image = abi.ImageBuffers(g.arr["xvals"], g.arr["yvals"], g.arr["data"], g.arr["mask"], c, 0.0)
    o = abi.srcgrid_defaults()
    for name, _t in abi.qlp_srcgrid_opts._fields_:
        setattr(o, name, getattr(g.opts, name))
    o.npixels_x, o.npixels_y = size
    o.regparam = lam
    r = O.evaluate(image, g.psf, o, g.lenses, regparam=0.0)
    N, M = r["n_active_pixels"], r["n_active_src"]
    L = O.get("Lpsf").reshape(-1, M)[:N].astype(np.longdouble)
    mask = g.arr["mask"].reshape(g.nx, g.ny)
    w = np.array([c[i, j] for j in range(g.ny) for i in range(g.nx) if mask[i, j]]).astype(np.longdouble)
    F = (L * w[:, None]).T @ L + np.longdouble(lam) * _curvature(O.get("active_index"), size)
    D = O.get("D")
    (La, neg), (Lb, _n) = _factor(F, np.longdouble), _factor(F, np.float64)
    assert neg
    la, lb = (2 * np.log(np.abs(np.diag(x))).sum() for x in (La, Lb))
    sa, sb = _solve(La, D), _solve(Lb, D)
    top = np.abs(sa).max()
    return (g, image, o, float(la), float(1e3 * abs(la - lb) + 1e-9 * abs(la)), sa.astype(float),
            float(1e3 * np.abs(sa - sb).max() + 1e-8 * top), F)


@pytest.mark.parametrize("size,lam,patch", CASES)
def test_reference_is_well_posed(size, lam, patch):
    _g, _i, _o, la, ltol, s, stol, F = _setup(size, lam, patch)
    assert np.isfinite(la) and ltol < 1e-6 * abs(la) and stol < 1e-4 * np.abs(s).max()
    rng, d = np.random.default_rng(0), np.sqrt(np.abs(np.diag(F)))
    for _ in range(4):
        E = np.tril(rng.uniform(-1, 1, F.shape))
        moved, _n = _factor(F + 2.0 ** -53 * (E + np.tril(E, -1).T) * np.outer(d, d), np.longdouble)
        assert abs(2 * np.log(np.abs(np.diag(moved))).sum() - la) < 0.1 * ltol


@pytest.mark.gpu
@pytest.mark.parametrize("size,lam,patch", CASES)
def test_goes_on_as_the_reference_does(size, lam, patch):
    from qlens_gb300 import PixelLikelihood, abi
    g, image, o, la, ltol, s, stol, _F = _setup(size, lam, patch)
    pl = PixelLikelihood.from_opts(image, g.psf, o, precision=abi.QLP_FP64)
    pl.set_lens_model(g.lenses, *g.zbeta())
    before = pl.invert_image_surface_brightness_map(regparam=10.0)
    r = pl.invert_image_surface_brightness_map()
    assert before["status"] == 0 and r["status"] == abi.QLP_ERR_NOT_SPD
    assert abs(r["logdet_F"] - la) <= ltol, (r["logdet_F"], la, ltol)
    assert np.abs(pl.dump(g.n_sub, r)["s"] - s).max() <= stol
    # its traces are gone from the next evaluations, and a batch gives the same
    after = pl.invert_image_surface_brightness_map(regparam=10.0)
    pl.set_batch_slots(2)
    batch = pl.eval_batch(np.array([g.params()] * 4), regparams=[10.0, 0.0, 0.0, 10.0])
    pl.close()
    for x in (after, batch[0], batch[3]):
        assert x["status"] == 0 and x["m2logev"] == before["m2logev"]
    for x in batch[1:3]:
        assert x["status"] == abi.QLP_ERR_NOT_SPD and x["logdet_F"] == r["logdet_F"] and x["chisq0"] == r["chisq0"]
