"""The elliptical NFW deflection's quadrature against the same nested rules in
extended precision, over scale radii that put the nodes below the tabulated
range of (xi/rs)^2 (QLens's logarithm), around 1 (its expansion), inside and
beyond it, for round to flat lenses and from loose to tight tolerances (few and
many levels of nodes), one lens and two.

Tolerance in u = 2^-53: a node's (xi/rs)^2 is within 6u, kappa's condition there
is at most 1 and its own error 2u, the factors add 5u; the sum over n nodes of
one sign (n + 1)u; the deflection's factors 4u.  Rays with a node where the
closed form itself loses digits (1e-5 <= |s - 1| < 2e-5) are left out."""
import os
import re

import numpy as np
import pytest

from goldens import Golden

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qlens_gb300", "csrc")


def _rule():
    text = open(os.path.join(CSRC, "patterson_rule.h")).read()
    out = []
    for name in ("QLP_PAT_POINTS_INIT", "QLP_PAT_WEIGHTS_INIT"):
        body = text[text.index("#define " + name):]
        body = body[body.index("{") + 1:body.index("}")]
        out.append(np.array([float(v) for v in re.findall(r"[-+0-9.e]+", body)]))
    return out


POINTS, WEIGHTS = _rule()


def _kappa(s):
    """kappa / ks with QLens's branches, in extended precision."""
    d = s - 1
    r = np.sqrt(np.abs(np.where(d == 0, 1, d)))
    F = np.where(d > 0, np.arctan(r), np.arctanh(np.where(d > 0, 0, np.minimum(r, 1 - np.longdouble(2) ** -60)))) / r
    near = np.abs(d) < 1e-5
    k = 2 * (1 - F) / np.where(near, 1, d)
    k = np.where(near, 2 * (np.longdouble(0.3333333333333333) - d / 5), k)
    return np.where(s < 1e-6, -(2 + np.log(s / 4)), k)


def _deflection(x, y, ks, rs, q, tol):
    """alpha, the nodes used, and whether a node lies where the closed form loses digits."""
    x, y = np.longdouble(x), np.longdouble(y)
    eps = 1 - np.longdouble(q) * np.longdouble(q)
    old, done, res, used, off, lossy = [0, 0], [False, False], [0, 0], [1, 1], 0, False
    for level in range(9):
        n = (2 << level) - 1
        i = (np.arange(n) + 1) * 2 ** (8 - level) - 1
        w = np.longdouble(0.5) + np.longdouble(0.5) * POINTS[i].astype(np.longdouble)
        wt = WEIGHTS[off:off + n].astype(np.longdouble)
        off += n
        u = w * w
        qf = 1 - eps * u
        s = u * (x * x + y * y / qf) * np.longdouble(q) / (np.longdouble(rs) * np.longdouble(rs))
        lossy |= bool(((np.abs(s - 1) > 0.99e-5) & (np.abs(s - 1) < 2e-5)).any())
        t = 2 * w * ks * _kappa(s) / np.sqrt(qf)
        for k, f in enumerate((t, t / qf)):
            if done[k]:
                continue
            res[k], used[k] = (wt * f).sum(), n
            if level > 1 and abs(res[k] - old[k]) < tol * abs(res[k]):
                done[k] = True
            old[k] = res[k]
        if all(done):
            break
    f = np.sqrt(1 - eps) * np.longdouble(0.5)
    return x * f * res[0], y * f * res[1], used, lossy


@pytest.mark.parametrize("rs", [2e-5, 3e-3, 0.7, 0.9, 40.0, 5e3])
@pytest.mark.parametrize("q,tol", [(0.999, 1e-3), (0.7, 1e-3), (0.25, 1e-3), (0.6, 1e-12)])
def test_deflection(rs, q, tol):
    from qlens_gb300 import PixelLikelihood, abi
    g = Golden("tiny_sie")
    pl = PixelLikelihood.from_opts(g.image, g.psf, g.opts, precision=abi.QLP_FP64)
    pl.set_nfw_tolerance(tol)
    ks = [0.4, 0.7]
    P = [[ks[0], rs, q, 0.0, 0.0, 0.0], [ks[1], rs, 1.0 - (1.0 - q) / 2, 0.0, 0.0, 0.0]]
    sets = []
    for n in (1, 2):
        pl.set_lens_model([{"type": "nfw", "plane": 0, "params": p} for p in P[:n]], [1.0], [[0.0]])
        r = pl.invert_image_surface_brightness_map(np.array(sum(P[:n], [])))
        sets.append(pl.dump(g.n_sub, r)["srcpt"].copy())
    # a lens of no mass: the rays' own positions
    pl.set_lens_model([{"type": "nfw", "plane": 0, "params": [0.0, 1.0, 1.0, 0.0, 0.0, 0.0]}], [1.0], [[0.0]])
    r = pl.invert_image_surface_brightness_map(np.array([0.0, 1.0, 1.0, 0.0, 0.0, 0.0]))
    pts = pl.dump(g.n_sub, r)["srcpt"].copy()
    pl.close()
    checked = 0
    for t in range(0, g.n_sub, max(1, g.n_sub // 60)):
        x, y = pts[2 * t], pts[2 * t + 1]
        ax = ay = np.longdouble(0)
        ex = ey = 4 * U
        lossy = False
        for n in range(2):
            # angle 0: the major axis along y, so the lens frame is (y, -x)
            dy, dx, used, bad = _deflection(y, -x, P[n][0], rs, P[n][2], tol)
            dx, used = -dx, used[::-1]
            lossy |= bad
            ax, ay = ax + dx, ay + dy
            ex += float(abs(dx)) * U * (18 + used[0])
            ey += float(abs(dy)) * U * (18 + used[1])
            if lossy:
                break
            got = sets[n][2 * t:2 * t + 2]
            scale = 3 * U * (max(abs(x), abs(y)) + float(max(abs(ax), abs(ay))))
            assert abs(float(x - ax - got[0])) <= ex + scale, (t, n, x, y)
            assert abs(float(y - ay - got[1])) <= ey + scale, (t, n, x, y)
            checked += 1
    assert checked > 20
