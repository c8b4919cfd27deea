"""The plain path's F = L'^T C^-1 L' + lambda R with noise maps of a wide range:
sqrt(C^-1) changing smoothly by 1e4 and 1e8 across the image (a step would leave F itself
too ill-conditioned to tell).  log det F against a factorisation in extended precision
of F summed in extended precision from the oracle's L'.

Tolerance: an FP64 sum of N terms and FP64 factorisation err by at most 4 N 2^-53
sqrt(F_ii F_jj) an entry, which moves log det F by at most 4 N 2^-53 M k, k the
condition number of F scaled to a unit diagonal (by numpy), and the oracle's L' itself has
(N_taps + 2) 2^-53 of each entry, within the same bound.
"""
import numpy as np
import pytest

from goldens import Golden

EPS = 2.0 ** -53
MAPS = [("x", 1e8), ("-y", 1e8), ("x", 1e4)]
SIZE = (9, 8)


def _covinv(g, kind):
    axis, ratio = kind
    t = np.arange(g.nx)[:, None] / (g.nx - 1.0) if axis == "x" else 1.0 - np.arange(g.ny)[None, :] / (g.ny - 1.0)
    s = 3.0 * ratio ** (t + np.zeros((g.nx, g.ny)))
    return s * s


def _curvature(ai, size):
    """R of the active cells (ai[j * nx + i], -1 inactive) from its definition Hx^T Hx + Hy^T Hy."""
    nx, ny = size
    ai = np.asarray(ai).reshape(ny, nx)
    M = int(ai.max()) + 1
    R = np.zeros((M, M))
    for dj, di in ((0, 1), (1, 0)):
        H = np.zeros((M, M))
        for j in range(ny):
            for i in range(nx):
                a = ai[j, i]
                if a < 0:
                    continue
                H[a, a] = -2
                for s in (-1, 1):
                    jj, ii = j + s * dj, i + s * di
                    if 0 <= jj < ny and 0 <= ii < nx and ai[jj, ii] >= 0:
                        H[a, ai[jj, ii]] = 1
        R += H.T @ H
    return R


def _logdet(F):
    """log det by an extended-precision Cholesky factorisation (in place)."""
    ld = 0
    A = F.copy()
    for k in range(len(A)):
        assert A[k, k] > 0
        A[k:, k] /= np.sqrt(A[k, k])
        A[k + 1:, k + 1:] -= np.outer(A[k + 1:, k], A[k + 1:, k])
        ld += 2 * np.log(A[k, k])
    return float(ld)


def _reference(g, kind, lam):
    """(log det F, its tolerance, the image) in extended precision."""
    from oracle import oracle as O
    from qlens_gb300 import abi
    c = _covinv(g, kind)
    image = abi.ImageBuffers(g.arr["xvals"], g.arr["yvals"], g.arr["data"], g.arr["mask"], c, 0.0)
    o = abi.srcgrid_defaults()
    for name, _t in abi.qlp_srcgrid_opts._fields_:
        setattr(o, name, getattr(g.opts, name))
    o.npixels_x, o.npixels_y = SIZE
    r = O.evaluate(image, g.psf, o, g.lenses, lens_params=np.array(g.params()), regparam=lam)
    assert r["status"] == 0
    N, M = r["n_active_pixels"], r["n_active_src"]
    L = O.get("Lpsf").reshape(-1, M)[:N].astype(np.longdouble)
    mask = g.arr["mask"].reshape(g.nx, g.ny)
    pix = [(i, j) for j in range(g.ny) for i in range(g.nx) if mask[i, j]]
    assert len(pix) == N                                       # every masked pixel is mapped
    w = np.array([c[p] for p in pix]).astype(np.longdouble)
    F = (L * w[:, None]).T @ L + np.longdouble(lam) * _curvature(O.get("active_index"), SIZE)
    d = np.sqrt(np.diag(F))
    k = np.linalg.cond((F / np.outer(d, d)).astype(float))
    return _logdet(F), 4 * N * EPS * M * k, o, image, r


@pytest.mark.parametrize("kind", MAPS)
def test_reference_is_well_posed(kind):
    """The tolerance is far below what lost digits move log det F by."""
    ref, tol, _o, _i, r = _reference(Golden("tiny_sie"), kind, 10.0)
    assert tol < 1e-3 and abs(r["logdet_F"] - ref) <= tol, (kind, ref, r["logdet_F"], tol)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", MAPS)
def test_logdet_matches_extended_precision(kind):
    from qlens_gb300 import PixelLikelihood, abi
    g = Golden("tiny_sie")
    ref, tol, o, image, _r = _reference(g, kind, 10.0)
    pl = PixelLikelihood.from_opts(image, g.psf, o, precision=abi.QLP_FP64)
    pl.set_lens_model(g.lenses, *g.zbeta())
    res = pl.invert_image_surface_brightness_map(regparam=10.0)
    batch = pl.eval_batch(np.array([g.params()] * 2), regparams=[10.0, 10.0])
    pl.close()
    assert res["status"] == 0
    assert abs(res["logdet_F"] - ref) <= tol, (kind, res["logdet_F"], ref, tol)
    assert all(b["status"] == 0 and b["logdet_F"] == res["logdet_F"] for b in batch)
