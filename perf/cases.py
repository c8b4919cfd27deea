"""Performance cases of the pixel likelihood, through the public Python interface.

Each case is work that a user of the library has it do: one likelihood
evaluation (what a simplex or Powell step, or looking at a reconstruction,
asks for), a batch of them (live points of a nested sampler, T-Walk
proposals), the fit drivers' likelihood with the regularisation parameter
optimised, and the training of the learned NFW deflection.  Sizes are those of
the repository's configurations (``qlens_gb300/synthetic.py``) and goldens, and
``draw`` spreads over the same ranges.

The inputs are made here: a Sersic source lensed by the case's own lens,
convolved with its PSF, plus seeded noise; the parameter vectors are drawn
around or over the prior box of the configuration that the case stands for.
``exact`` is the same likelihood in plain FP64 torch.
"""
import math

import numpy as np
import torch

from qlens_gb300 import PixelLikelihood, abi
from qlens_gb300 import pixlike

# A likelihood's value and its terms, as qlp_result names them, and its counts.
VALUES = ("m2logev", "chisq0", "logdet_F", "logdet_R", "Es_times_two", "regterms")
COUNTS = ("n_active_pixels", "n_active_src", "L_nnz", "status")

# Two lens planes (z = 0.5 and 0.8, source at z = 2) and the subhalo's
# cosmology (sigma_cr, kpc to arcsec, critical density), as the goldens hold them.
ZFAC = [1.0, 1.0]
BETA = [[0.50757349]]
COSMO = [131218470966.34126, 0.13318529787886016, 333084360000.0]

# The learned NFW deflection that the subhalo cases use: a short training
# (the subhalo's deflections are small, so its error bound passes the gate).
SURROGATE = dict(n_train=1 << 18, batch=16384, steps=3000)
_trained = {"opts": None}       # what the process's surrogate was last trained with


def _case(name, kind, precision, lens, nx, ny, pixel, rin, rout, nsplit, psf, src, n=1, uneven=False, noise=0.02,
          lam=10.0, recon=False):
    return dict(name=name, kind=kind, precision=precision, lens=lens, nx=nx, ny=ny, pixel=pixel, rin=rin, rout=rout,
                nsplit=nsplit, psf_x=psf[0], psf_y=psf[1], src_x=src[0], src_y=src[1], n=n, uneven=uneven,
                noise=noise, lam=lam, recon=recon)


def listed():
    return [
        # the smallest use: a postage stamp, one evaluation and its source and
        # model image, as when a model is set up and looked at
        _case("stamp_fp64", "single", "fp64", "sie", 24, 24, 0.1, 0.0, 1.2, 3, (5, 5), (10, 10), noise=0.03, lam=5.0,
              recon=True),
        # the reference's own case, evaluated one at a time (simplex, Powell)
        _case("small_fp64", "single", "fp64", "sie", 80, 80, 0.05, 0.0, 2.5, 2, (7, 7), (30, 30), recon=True),
        # the same image under a sampler: 32 proposals a call
        _case("small_mixed_b32", "batch", "mixed", "sie", 80, 80, 0.05, 0.0, 2.5, 2, (7, 7), (30, 30), n=32),
        # a space-telescope image, power law, 64x64 source: one exact evaluation
        _case("large_fp64", "single", "fp64", "power", 200, 200, 0.04, 0.5, 2.5, 4, (21, 21), (64, 64), noise=0.01),
        # ... one evaluation of the mixed path (its latency)
        _case("large_mixed", "single", "mixed", "power", 200, 200, 0.04, 0.5, 2.5, 4, (21, 21), (64, 64), noise=0.01),
        # ... and 32 at once (its throughput)
        _case("large_mixed_b32", "batch", "mixed", "power", 200, 200, 0.04, 0.5, 2.5, 4, (21, 21), (64, 64), n=32,
              noise=0.01),
        # nested-sampling live points: every vector its own mask, source grid and lambda
        _case("uneven_mixed_b128", "batch", "mixed", "sie", 100, 100, 0.05, 0.0, 3.0, 2, (11, 11), (64, 64), n=128,
              uneven=True),
        # the same live points on the exact path, fewer of them
        _case("uneven_fp64_b16", "batch", "fp64", "sie", 100, 100, 0.05, 0.0, 3.0, 2, (11, 11), (64, 64), n=16,
              uneven=True),
        # an elliptical NFW halo by the adaptive quadrature, the whole frame masked in
        _case("halo_mixed_b8", "batch", "mixed", "nfw", 200, 200, 0.04, 0.0, 4.5, 4, (21, 21), (48, 48), n=8,
              noise=0.01),
        # two planes with a subhalo through the learned deflection, uneven grids: the
        # configuration of the headline benchmark, one wave of its batch
        _case("subhalo_mixed_b32", "batch", "mixed", "subhalo", 300, 300, 0.03, 0.3, 3.5, 4, (31, 31), (64, 64), n=32,
              uneven=True, noise=0.1),
        # the fit drivers' likelihood with lambda optimised, an odd-sized real image's shape
        _case("fit_lambda_fp64_b4", "fit", "fp64", "power", 81, 81, 0.049, 0.6, 1.9, 2, (7, 9), (40, 40), n=4,
              noise=0.01, lam=20.0),
        # training the learned deflection (forward and backward), shortened
        dict(name="train_surrogate", kind="train", n_train=1 << 17, batch=16384, steps=256),
    ]


def _seconds(c):
    """A rough time of a case, to keep the drawn ones within the listed ones."""
    if c["kind"] == "train":
        return 0.3 * c["steps"] / 256.0 * c["batch"] / 16384.0
    N, M, rays = _sizes(c)
    one = rays * (4e-9 if c["lens"] in ("nfw", "subhalo") and c["precision"] == "fp64" else 1.5e-9)
    if c["precision"] == "fp64":
        one += 0.25e-12 * N * M * M + 1.8e-12 * M ** 3 + 6e-6 * M + 3e-10 * N * c["psf_x"] * c["psf_y"]
    else:
        one += 2e-15 * N * M * M + 1e-14 * M ** 3 + 5e-11 * N * c["psf_x"] * c["psf_y"] + 1e-4
    if c["kind"] == "single":
        one += 1e-6 * M
    if c["kind"] == "fit":
        one *= 6
    return one * c["n"]


def draw(rng):
    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    def odd(a, b):
        return 2 * (int(round(log(a, b))) // 2) + 1

    while True:
        what = rng.random()
        if what < 0.06:
            c = dict(kind="train", n_train=1 << rng.randint(16, 18), batch=256 * int(log(16, 64)),
                     steps=int(log(32, 256)))
        else:
            kind = "single" if what < 0.45 else "batch" if what < 0.85 else "fit"
            precision = "fp64" if kind == "fit" or rng.random() < 0.5 else "mixed"
            lens = rng.choice(["sie", "sie", "power", "power", "nfw", "subhalo"])
            if kind == "fit":
                lens = rng.choice(["sie", "power"])
            nx = int(round(log(20, 300)))
            ny = max(20, min(300, int(round(nx * rng.uniform(0.85, 1.2)))))
            rout = rng.uniform(1.6, 3.5)
            # the frame spans the mask, more or less
            pixel = 2.0 * rout / min(nx, ny) * rng.uniform(0.85, 1.4)
            big = max(3, min(31, min(nx, ny) // 3))
            src = int(round(log(8, 64)))
            c = _case("", kind, precision, lens, nx, ny, pixel, rng.choice([0.0, 0.0, 0.3, 0.6]), rout,
                      rng.choice([2, 2, 3, 4]), (odd(3, big), odd(3, big)),
                      (src, max(6, min(64, src + rng.randint(-3, 3)))),
                      n=1 if kind == "single" else int(round(log(2, 4 if kind == "fit" else 96))),
                      uneven=kind == "batch" and rng.random() < 0.5,
                      noise=log(0.01, 0.1), lam=log(3.0, 50.0), recon=kind == "single" and rng.random() < 0.5)
            del c["name"]
        if 2e-4 < _seconds(c) < 0.08:
            return c


# ---- inputs ----------------------------------------------------------------
def _axis(n, pixel):
    step = (n * pixel) / n
    return np.array([-0.5 * n * pixel + i * step for i in range(n + 1)])


def _mask(xv, yv, rin, rout):
    x, y = 0.5 * (xv[:-1] + xv[1:]), 0.5 * (yv[:-1] + yv[1:])
    rsq = x[:, None] ** 2 + y[None, :] ** 2
    return ((rsq >= rin * rin) & (rsq < rout * rout)).astype(np.uint8)


def _psf(c):
    """A core with wings, positive at every tap, unit sum."""
    x = np.arange(c["psf_x"]) - c["psf_x"] // 2
    y = np.arange(c["psf_y"]) - c["psf_y"] // 2
    a = 0.2 * max(3, min(c["psf_x"], c["psf_y"]))
    v = (1 + (x[:, None] ** 2 + y[None, :] ** 2) / a ** 2) ** -2.0
    return v / v.sum()


def _sizes(c):
    """(masked pixels, source cells in use, rays) of one evaluation; uneven batches: of their mean."""
    xv, yv = _axis(c["nx"], c["pixel"]), _axis(c["ny"], c["pixel"])
    N = int(_mask(xv, yv, c["rin"], c["rout"]).sum())
    M = 0.75 * c["src_x"] * c["src_y"]
    if c["uneven"]:
        M *= 0.55
        N = int(0.7 * N) if c["lens"] != "subhalo" else N
    return N, M, N * c["nsplit"] ** 2


def _lenses(kind, p):
    """The lens list with one parameter vector's values as its defaults."""
    spec = [dict(type="sple", params=list(p[:7])), dict(type="shear", params=list(p[7:11]))]
    if kind == "nfw":
        spec.append(dict(type="nfw", params=list(p[11:17])))
    elif kind == "subhalo":
        spec.append(dict(type="nfw_m200_c", params=list(p[11:17]), plane=1, cosmo=COSMO))
    return spec


def _truth(c):
    p = [1.2, 1.05 if c["lens"] == "power" else 1.0, 0.0, 0.8, 30.0, 0.0, 0.0, 0.05, 10.0, 0.0, 0.0]
    if c["lens"] == "nfw":
        p += [0.05, 8.0, 0.8, 20.0, 0.05, -0.05]
    elif c["lens"] == "subhalo":
        p += [1e9, 10.0, 0.8, 0.0, 0.9, 0.6]
    return np.array(p)


def _draws(c, rng):
    """n parameter vectors: the prior box of the configuration, for the subhalo the posterior region."""
    n, P = c["n"], np.tile(_truth(c), (c["n"], 1))
    if c["lens"] == "subhalo":
        for i, s in {0: 2e-5, 3: 6e-5, 4: 2e-3, 7: 4e-5, 8: 1e-2, 11: 5e6, 12: 0.12, 13: 5e-3, 14: 2.0, 15: 2e-3,
                     16: 1e-3}.items():
            P[:, i] += 3.0 * s * rng.uniform(-1.0, 1.0, n)
        return P
    P[:, 0] = rng.uniform(1.0, 1.4, n)
    P[:, 3] = rng.uniform(0.6, 0.95, n)
    P[:, 4] = rng.uniform(0.0, 180.0, n)
    P[:, 7] = rng.uniform(0.0, 0.1, n)
    P[:, 8] = rng.uniform(0.0, 180.0, n)
    if c["lens"] == "power":
        P[:, 1] = rng.uniform(0.9, 1.2, n)
    elif c["lens"] == "sie":
        P[:, 5] = P[:, 9] = rng.uniform(-0.1, 0.1, n)
        P[:, 6] = P[:, 10] = rng.uniform(-0.1, 0.1, n)
    elif c["lens"] == "nfw":
        P[:, 11] = rng.uniform(0.05, 0.5, n)
        P[:, 12] = rng.uniform(2.0, 20.0, n)
        P[:, 13] = rng.uniform(0.5, 1.0, n)
        P[:, 14] = rng.uniform(0.0, 180.0, n)
    return P


# The fit drivers' parameters: b and the axis ratio with Gaussian priors, the
# angle, the shear by its logarithm.
FIT = [dict(target=0, prior=abi.QLP_PRIOR_GAUSS, prior_pos=1.2, prior_sig=0.2, prior_norm=1.0),
       dict(target=3, prior=abi.QLP_PRIOR_GAUSS, prior_pos=0.8, prior_sig=0.1, prior_norm=1.0),
       dict(target=4), dict(target=7, transform=abi.QLP_TRANSFORM_LOG, include_jacobian=1)]


def _inputs(c, seed):
    """Everything that the case's call is given, as numpy arrays."""
    rng = np.random.default_rng(seed)
    xv, yv = _axis(c["nx"], c["pixel"]), _axis(c["ny"], c["pixel"])
    psf = _psf(c)
    sharp = torch.zeros((c["nx"], c["ny"]), dtype=torch.float64, device="cuda")
    truth = _truth(c)
    for sx, sy in ((0.25, 0.25), (0.25, 0.75), (0.75, 0.25), (0.75, 0.75)):
        x = torch.as_tensor((1 - sx) * xv[:-1] + sx * xv[1:], device="cuda")
        y = torch.as_tensor((1 - sy) * yv[:-1] + sy * yv[1:], device="cuda")
        bx, by = _source_points(c["lens"], truth, *torch.meshgrid(x, y, indexing="ij"))
        sharp += 0.25 * _sersic(bx, by)
    img = torch.zeros_like(sharp)
    hx, hy = c["psf_x"] // 2, c["psf_y"] // 2
    pad = torch.nn.functional.pad(sharp, (hy, hy, hx, hx))
    for k in range(c["psf_x"]):
        for l in range(c["psf_y"]):
            img += psf[k, l] * pad[2 * hx - k:2 * hx - k + c["nx"], 2 * hy - l:2 * hy - l + c["ny"]]
    data = img.cpu().numpy() + c["noise"] * rng.standard_normal((c["nx"], c["ny"]))
    P = _draws(c, rng)
    d = dict(xv=xv, yv=yv, psf=psf, data=data, mask=_mask(xv, yv, c["rin"], c["rout"]), P=P, lam=None, masks=None,
             mask_ids=None, sizes=None)
    if c["uneven"]:
        n = c["n"]
        sx = rng.integers(max(6, c["src_x"] // (2 if c["lens"] == "subhalo" else 3)), c["src_x"] + 1, n)
        d["sizes"] = np.stack([sx, np.minimum(sx, c["src_y"])], 1)
        if c["lens"] != "subhalo":
            radii = rng.uniform(0.5 * (c["rin"] + c["rout"]), c["rout"], min(n, 64))
            d["masks"] = np.stack([_mask(xv, yv, c["rin"], r).ravel() for r in radii])
            d["mask_ids"] = rng.integers(0, len(radii), n)
            d["lam"] = 10.0 ** rng.uniform(0.5, 2.0, n)
    return d


def prepare(case, seed):
    if case["kind"] == "train":
        # points of the trained domain at which the caller looks at the network
        rng = np.random.default_rng(seed)
        points = np.stack([rng.uniform(math.log(1e-3), math.log(100.0), 4096), rng.uniform(0.0, math.pi / 2, 4096),
                           rng.uniform(0.5, 0.99, 4096)], 1)
        return dict(case=case, seed=int(seed) % 1000 + 1, points=points)
    d = _inputs(case, seed)
    pl = PixelLikelihood(d["xv"], d["yv"], d["data"], d["mask"], d["psf"], bg_noise=case["noise"],
                         nsplit=case["nsplit"], src_npixels=(case["src_x"], case["src_y"]), regparam=case["lam"],
                         precision=abi.QLP_MIXED if case["precision"] == "mixed" else abi.QLP_FP64)
    two = case["lens"] == "subhalo"
    pl.set_lens_model(_lenses(case["lens"], d["P"][0]), ZFAC if two else None, BETA if two else None)
    if two and case["precision"] == "mixed":
        if _trained["opts"] != SURROGATE:
            pixlike.train_nfw_surrogate(**SURROGATE)
            _trained["opts"] = SURROGATE
        pl.set_nfw_mode(abi.QLP_NFW_SURROGATE)
    if case["kind"] != "single":
        pl.set_batch_slots(min(case["n"], 32))
    if d["masks"] is not None:
        pl.set_instance_masks(d["masks"])
    s = dict(case=case, pl=pl, **d)
    if case["kind"] == "fit":
        pl.set_fit_params(FIT)
        pl.set_regparam_optimization(True)
        s["X"] = np.stack([d["P"][:, 0], d["P"][:, 3], d["P"][:, 4],
                           np.log10(np.maximum(d["P"][:, 7], 1e-3))], 1)
    return s


# ---- the calls ---------------------------------------------------------------
def run(state):
    c = state["case"]
    if c["kind"] == "train":
        _trained["opts"] = None
        r = pixlike.train_nfw_surrogate(n_train=c["n_train"], batch=c["batch"], steps=c["steps"], seed=state["seed"])
        t, _, _, bound = pixlike.surrogate_eval(state["points"])
        return dict({k: np.float32(r[k]) for k in ("final_loss", "val_max_rel", "val_mean_rel", "cells_below_1e5")},
                    net=t.astype(np.float32), bound=bound.astype(np.float32))
    pl = state["pl"]
    # the exact path's results are FP64; the mixed path's hang on an FP32 factor
    real = np.float64 if c["precision"] == "fp64" else np.float32
    out = {}
    if c["kind"] == "single":
        res = [pl.invert_image_surface_brightness_map(state["P"][0], c["lam"])]
        if c["recon"]:
            n_mask = int(state["mask"].sum())
            d = pl.dump(n_mask * c["nsplit"] ** 2, res[0])
            # on the whole source grid, and on the mask's pixels
            used = d["active_index"] >= 0
            for k in ("D", "s"):
                out[k] = np.zeros(c["src_x"] * c["src_y"], real)
                out[k][used] = d[k][d["active_index"][used]]
            out["model"] = np.zeros(n_mask, real)
            out["model"][:res[0]["n_active_pixels"]] = d["model"]
    elif c["kind"] == "batch":
        res = pl.eval_batch(state["P"], state["lam"], state["mask_ids"], state["sizes"])
    else:
        ll, res = pl.fit_loglike_batch(state["X"])
        out["loglike"] = np.asarray(ll, real)
        out["regparam"] = np.array([r["regparam"] for r in res], real)
    out.update({k: np.array([r[k] for r in res], real) for k in VALUES})
    out.update({k: np.array([r[k] for r in res], np.int64) for k in COUNTS})
    return out


def work(case):
    if case["kind"] == "train":
        # forward and backward of the 3 -> 4 x 128 -> 2 network: 6 operations a weight and sample
        return {"bytes": 20.0 * case["n_train"], "flops": 6.0 * 50306 * case["batch"] * case["steps"]}
    N, M, rays = _sizes(case)
    taps = case["psf_x"] * case["psf_y"]
    n = case["n"]
    # image, inverse variance, mask and PSF once; a vector and a result per evaluation
    given = case["nx"] * case["ny"] * 17.0 + 8.0 * taps + n * (8.0 * 17 + 8.0 * len(VALUES) + 4.0 * len(COUNTS))
    # rays, the PSF on L (3 entries a ray at most, merged to about 10 a pixel),
    # the lower triangle of F dense, F's factor, R's banded factor, the solve
    one = 60.0 * rays + 2.0 * taps * 10 * N + N * M * M + M ** 3 / 3.0 + M * (2.0 * case["src_x"]) ** 2 + 4.0 * M * M
    if case["kind"] == "fit":
        one += 9 * (M ** 3 / 3.0 + 4.0 * M * M + 4.0 * N * M)       # about ten trials of lambda
    if case["recon"]:
        given += 8.0 * (2 * M + N)
    return {"bytes": given, "flops": n * one}


# ---- the same in plain FP64 torch --------------------------------------------
def _rotate(x, y, theta_deg):
    th = math.radians(theta_deg)
    c, s = -math.sin(th), math.cos(th)
    return x * c + y * s, y * c - x * s, c, s


def _sple(p, x, y):
    b, alpha, _, q, theta, xc, yc = (float(v) for v in p)
    X, Y, c, s = _rotate(x - xc, y - yc, theta)
    bp = b / math.sqrt(q)
    if alpha == 1.0:
        psi, u = torch.sqrt(q * q * X * X + Y * Y), math.sqrt(1 - q * q)
        ax, ay = bp * q / u * torch.atan(u * X / psi), bp * q / u * torch.atanh(u * Y / psi)
    else:
        # the angular series of an elliptical power law (Tessore & Metcalf 2015)
        R, phi = torch.sqrt(X * X + Y * Y / (q * q)), torch.atan2(Y / q, X)
        f, beta = (1 - q) / (1 + q), 2.0 / (2.0 - alpha)
        term = torch.polar(torch.ones_like(phi), phi)
        turn = torch.polar(torch.ones_like(phi), 2 * phi)
        total = term.clone()
        for i in range(1, 90):
            term = term * turn * (-f * (beta * i - 1) / (beta * i + 1))
            total += term
        scale = 2 * bp * q / (1 + q) * (bp / R) ** (alpha - 1)
        ax, ay = scale * total.real, scale * total.imag
    return ax * c - ay * s, ax * s + ay * c


def _nfw(ks, rs, q, theta, xc, yc, x, y):
    X, Y, c, s = _rotate(x - xc, y - yc, theta)
    t, wt = np.polynomial.legendre.leggauss(96)
    i0, i1 = torch.zeros_like(X), torch.zeros_like(X)
    for a, w in zip(0.5 + 0.5 * t, 0.5 * wt):
        qf = 1 - (1 - q * q) * a * a
        z = a * a * q * (X * X + Y * Y / qf) / (rs * rs)
        r = torch.sqrt((z - 1).abs()).clamp_min(1e-12)
        g = torch.where(z > 1, torch.atan(r), torch.atanh(r.clamp_max(1 - 1e-16))) / r
        near = (z - 1).abs() < 1e-5
        kap = torch.where(near, 2 * ks * (1.0 / 3 - (z - 1) / 5), 2 * ks * (1 - g) / torch.where(near, 1.0, z - 1))
        f = 2 * a * w / math.sqrt(qf) * kap
        i0 += f
        i1 += f / qf
    ax, ay = q * X * i0, q * Y * i1
    return ax * c - ay * s, ax * s + ay * c


def _source_points(kind, p, x, y):
    """The lens equation for the image points (x, y)."""
    ax, ay = _sple(p[:7], x, y)
    te = math.radians(p[8]) + 0.5 * math.pi
    g1, g2 = p[7] * math.cos(2 * te), p[7] * math.sin(2 * te)
    dx, dy = x - p[9], y - p[10]
    ax, ay = ax + dx * g1 + dy * g2, ay - dy * g1 + dx * g2
    if kind == "nfw":
        hx, hy = _nfw(*(float(v) for v in p[11:17]), x, y)
        ax, ay = ax + hx, ay + hy
    elif kind == "subhalo":
        m, c200, q, theta, xc, yc = (float(v) for v in p[11:17])
        sigma_cr, kpc, crit = COSMO
        rs = (m / (200 * 4 * math.pi / 3 * 1e-9 * crit)) ** (1.0 / 3) / c200 * kpc
        ks = m / (4 * math.pi * rs * rs * sigma_cr * (math.log(1 + c200) - c200 / (1 + c200)))
        hx, hy = _nfw(ks, rs, q, theta, xc, yc, x - BETA[0][0] * ax, y - BETA[0][0] * ay)
        ax, ay = ax + hx, ay + hy
    return x - ax, y - ay


def _sersic(bx, by, reff=0.2, n=1.5, q=0.75, theta=20.0, xc=0.04, yc=-0.02):
    th = math.radians(theta)
    dx, dy = bx - xc, by - yc
    u, v = dx * math.cos(th) + dy * math.sin(th), -dx * math.sin(th) + dy * math.cos(th)
    bn = 2 * n - 1.0 / 3 + 4.0 / (405 * n)
    return torch.exp(-bn * ((torch.sqrt(q * u * u + v * v / q) / reff) ** (1.0 / n) - 1))


def _grid(means, n):
    """Corners and centres of the source grid along one axis, from the per-pixel mean source points."""
    lo, hi = float(means.min()), float(means.max())
    w = 0.1 * (hi - lo)
    lo, hi = lo - w / 2, hi + w / 2
    corner = np.add.accumulate(np.concatenate([[lo], np.full(n, (hi - lo) / n)]))
    corner = torch.as_tensor(corner, device="cuda")
    return corner, (corner[:-1] + corner[1:]) / 2


def _axis_cells(p, corner, centre):
    n = len(centre)
    i = (torch.searchsorted(corner, p.contiguous(), right=True) - 1).clamp(0, n - 1)
    up = ((p > centre[i]) & (i < n - 1)) | (i == 0)
    return i, torch.where(up, i + 1, i - 1)


def _likelihood(c, d, p, lam, mask, snx, sny):
    """One evaluation: the values by name, and D, s and the model image."""
    cu = dict(device="cuda")
    nx, ny, ns = c["nx"], c["ny"], c["nsplit"]
    pj, pi = np.nonzero(mask.reshape(nx, ny).T)          # j outer, i inner
    pi, pj = torch.as_tensor(pi, **cu), torch.as_tensor(pj, **cu)
    xv, yv = torch.as_tensor(d["xv"], **cu), torch.as_tensor(d["yv"], **cu)
    u = (1.0 + 2.0 * torch.arange(ns, dtype=torch.float64, **cu)) / (2 * ns)
    x = (xv[pi, None] * (1 - u) + xv[pi + 1, None] * u)[:, :, None].expand(-1, ns, ns)
    y = (yv[pj, None] * (1 - u) + yv[pj + 1, None] * u)[:, None, :].expand(-1, ns, ns)
    bx, by = _source_points(c["lens"], p, x.reshape(len(pi), -1), y.reshape(len(pi), -1))
    cx, ccx = _grid(bx.mean(1), snx)
    cy, ccy = _grid(by.mean(1), sny)
    inside = (bx >= cx[0]) & (bx < cx[-1]) & (by >= cy[0]) & (by < cy[-1])
    i, i2 = _axis_cells(bx, cx, ccx)
    j, j2 = _axis_cells(by, cy, ccy)
    # the three cells of the interpolation and their barycentric weights
    fx, fy = (bx - ccx[i]) / (ccx[i2] - ccx[i]), (by - ccy[j]) / (ccy[j2] - ccy[j])
    cells = torch.stack([j * snx + i, j * snx + i2, j2 * snx + i], -1)
    w = torch.stack([1 - fx - fy, fx, fy], -1) / (ns * ns) * inside[..., None]
    used = torch.zeros(snx * sny, dtype=torch.bool, **cu)
    used[cells[inside].reshape(-1)] = True
    M = int(used.sum())
    index = torch.cumsum(used, 0) - 1
    rows = inside.any(1)
    N = int(rows.sum())
    L = torch.zeros((N + 1, M), dtype=torch.float64, **cu)      # the last row stays zero
    at = torch.arange(N, **cu)[:, None, None].expand(N, ns * ns, 3)
    keep = inside[rows][..., None].expand(N, ns * ns, 3)
    L.index_put_((at[keep], index[cells[rows][keep]]), w[rows][keep], accumulate=True)
    where = torch.full((nx + 2 * c["psf_x"], ny + 2 * c["psf_y"]), N, dtype=torch.int64, **cu)
    ri, rj = pi[rows] + c["psf_x"], pj[rows] + c["psf_y"]
    where[ri, rj] = torch.arange(N, **cu)
    Lp = torch.zeros((N, M), dtype=torch.float64, **cu)
    for k in range(c["psf_x"]):
        for l in range(c["psf_y"]):
            Lp.add_(L[where[ri + c["psf_x"] // 2 - k, rj + c["psf_y"] // 2 - l]], alpha=float(d["psf"][k, l]))
    del L
    cinv = 1.0 / (c["noise"] * c["noise"])
    data = torch.as_tensor(d["data"], **cu)[pi, pj]
    D = Lp.T @ data[rows] * cinv
    F = Lp.T @ Lp * cinv
    # curvature: (-2 at a cell, 1 at each active neighbour) along x, and along y
    R = torch.zeros((M, M), dtype=torch.float64, **cu)
    ids = torch.where(used, index, M).reshape(sny, snx)
    for dy, dx in ((0, 1), (1, 0)):
        H = torch.zeros((M, M + 1), dtype=torch.float64, **cu)
        me = torch.arange(M, **cu)
        H[me, me] = -2.0
        for sign in (1, -1):
            pad = torch.full((sny + 2, snx + 2), M, dtype=torch.int64, **cu)
            pad[1:-1, 1:-1] = ids
            near = pad[1 + sign * dy:1 + sign * dy + sny, 1 + sign * dx:1 + sign * dx + snx].reshape(-1)[used]
            H[me, near] = 1.0
        H = H[:, :M]
        R += H.T @ H
        del H
    F = torch.linalg.cholesky(F.add_(R, alpha=lam))
    s = torch.cholesky_solve(D[:, None], F)[:, 0]
    ldF = 2 * float(torch.log(torch.diagonal(F)).sum())
    ldR = 2 * float(torch.log(torch.diagonal(torch.linalg.cholesky(R))).sum())
    model = torch.zeros(len(pi), dtype=torch.float64, **cu)
    model[:N] = Lp @ s
    chi = float(((model[:N] - data[rows]) ** 2).sum() + (data[~rows] ** 2).sum()) * cinv
    es = float(s @ (R @ s))
    reg = lam * es - M * math.log(lam) - ldR
    source = torch.zeros((2, snx * sny), dtype=torch.float64, **cu)
    source[0][used], source[1][used] = D, s
    return dict(m2logev=chi + reg + ldF, chisq0=chi, logdet_F=ldF, logdet_R=ldR, Es_times_two=es, regterms=reg,
                D=source[0], s=source[1], model=model)


def exact(case, seed):
    # lambda is where a search with a tolerance stops, and a training's result is
    # where its rounding took it: neither has a value in 64 bits
    if case["kind"] in ("fit", "train"):
        return None
    N, M, rays = _sizes(case)
    one = 3e-12 * N * M * M + 1.2e-11 * case["psf_x"] * case["psf_y"] * N * M + 4e-12 * M ** 3
    one += 2e-6 * rays if case["lens"] in ("nfw", "subhalo") else 0.0
    if case["n"] * (one + 0.02) > 22.0:
        return None
    d = _inputs(case, seed)
    got = []
    for v in range(case["n"]):
        mask = d["mask"] if d["masks"] is None else d["masks"][d["mask_ids"][v]]
        size = (case["src_x"], case["src_y"]) if d["sizes"] is None else (int(d["sizes"][v][0]), int(d["sizes"][v][1]))
        got.append(_likelihood(case, d, d["P"][v], case["lam"] if d["lam"] is None else float(d["lam"][v]), mask, *size))
    out = {k: np.array([g[k] for g in got]) for k in VALUES}
    out.update({k: None for k in COUNTS})
    if case["recon"]:
        out.update({k: got[0][k].cpu().numpy() for k in ("D", "s", "model")})
    return out
