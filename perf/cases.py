"""The work that is timed: what a program that fits galaxies with this package has it do.

A fit evaluates chi2 and its gradient for one proposal after another on a
packed patch (``evaluate``, ``residual``, ``forward``, ``autograd``), on many
patches or chains at once (``batch``, ``chains``), solves the linear fluxes of
fixed shapes (``flux``) and packs its patches from exposures held in device
memory (``pack``).  Sizes are those of this repository's workloads (one source
on 64 x 64 pixels; 20 sources in 8 bands x 4 exposures; 60 sources in 15 bands
x 6 exposures; uneven patches of 32 to 200 pixels a side; 2048 x 2048
exposures in 8 x 8 super-pixels) and sizes between them.

Patches come from :mod:`forcepho_b200.synth`; their truth images are rendered
here in 64 bits.  ``exact`` evaluates the same quantities in 64 bits with torch
alone, from the packed arrays.
"""

import math

import numpy as np
import torch

from forcepho_b200 import synth
from forcepho_b200.autograd import PatchEvaluator, lnlike
from forcepho_b200.batch import PatchBatch
from forcepho_b200.device_proposal import DeviceSersicTable, SOURCE_BYTES
from forcepho_b200.fitting import optimize_fluxes_device
from forcepho_b200.patches.device_store import REGION_DTYPE, DeviceStore
from forcepho_b200.proposal import GPUProposer
from forcepho_b200.region import REGION_CIRCLE, RectangularRegion
from forcepho_b200.sampling import ChainCopy
from forcepho_b200.sources import default_table, proposal_from_params
from forcepho_b200.wcs import TanWCS

F64 = dict(dtype=torch.float64, device="cuda")
CUTOFF = 36.0        # a Gaussian's exp-argument beyond which it is not evaluated
N_RADII = 9          # mixture radii of the packaged Sersic table
PAIRS_MAX = 60 * 54 * 90 * 256 * 256   # (pixel, Gaussian) pairs of the largest listed patch


# ------------------------------------------------------------------ the cases
def listed():
    def patch(name, kind, ns, nb, ne, nx, ny, n_psf, order):
        return dict(name=name, kind=kind, n_sources=ns, n_bands=nb, n_exp=ne, nx=nx, ny=ny,
                    n_psf=n_psf, order=order)

    return [
        # the smallest call: one isolated galaxy, one exposure, results on the host
        patch("one_source", "evaluate", 1, 1, 1, 64, 64, 3, "morton"),
        # an ordinary small patch, its pixels in the order of a pixel store
        patch("small_patch", "evaluate", 3, 2, 3, 56, 48, 3, "store"),
        # the benchmark's patch: 20 sources, 8 bands x 4 exposures
        patch("field", "evaluate", 20, 8, 4, 128, 128, 5, "morton"),
        # the largest patch: 60 sources, 15 bands x 6 exposures
        patch("crowded", "evaluate", 60, 15, 6, 256, 256, 6, "store"),
        # subtraction of sources: the residual image comes back too; ragged stamps
        patch("residual", "residual", 7, 3, 2, 97, 83, 4, "morton"),
        # the likelihood without its gradient, on the device (line searches, Metropolis tests)
        patch("forward", "forward", 12, 5, 3, 120, 112, 5, "store"),
        # gradient descent: single-precision parameters through torch autograd
        patch("autograd", "autograd", 10, 4, 4, 100, 100, 4, "morton"),
        # a mosaic's patches advanced together, uneven as they come
        dict(name="batch", kind="batch", n_patches=48, max_sources=30, max_bands=8, max_exp=8,
             max_side=200, n_psf=5, layout=0),
        # many chains of one small patch: proposals from parameters, then one batched evaluation
        dict(name="chains", kind="chains", n_chains=256, n_sources=1, n_bands=1, n_exp=1, nx=64,
             ny=64, n_psf=3),
        # fluxes and their precision at fixed shapes, from the scene to the solution
        patch("flux", "flux", 20, 8, 4, 128, 128, 5, "morton"),
        # one patch's pixels out of exposures resident in device memory
        dict(name="pack_one", kind="pack", side=2048, n_exp=32, n_patches=1, radius=68.0,
             shape="circle", background=True, max_snr=0.0, layout=0),
        # the pixels of 32 patches in one call, with the signal-to-noise cap
        dict(name="pack_many", kind="pack", side=2048, n_exp=32, n_patches=32, radius=68.0,
             shape="circle", background=True, max_snr=100.0, layout=1),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "evaluate", "residual", "forward", "autograd",
                       "batch", "chains", "flux", "pack"])
    if kind == "batch":
        return dict(kind=kind, n_patches=int(_log(rng, 8, 48)), max_sources=rng.randint(4, 30),
                    max_bands=rng.randint(1, 8), max_exp=rng.randint(1, 8),
                    max_side=rng.randint(48, 200), n_psf=rng.randint(3, 5),
                    layout=rng.randrange(1000))
    if kind == "chains":
        return dict(kind=kind, n_chains=int(_log(rng, 16, 300)), n_sources=rng.randint(1, 2),
                    n_bands=rng.randint(1, 3), n_exp=rng.randint(1, 2), nx=rng.randint(40, 72),
                    ny=rng.randint(40, 72), n_psf=rng.randint(2, 4))
    if kind == "pack":
        n = int(_log(rng, 1, 32))
        return dict(kind=kind, side=rng.choice([512, 1024, 2048]), n_exp=rng.randint(4, 32),
                    n_patches=n, radius=round(rng.uniform(20.0, 80.0), 2),
                    shape="circle" if n > 4 or rng.random() < 0.7 else "box",
                    background=rng.random() < 0.5, max_snr=rng.choice([0.0, 100.0]),
                    layout=rng.randrange(1000))
    order = rng.choice(["morton", "store"])
    side_max = 256 if kind == "evaluate" else 200
    while True:
        ns = int(_log(rng, 1, 60 if kind == "evaluate" else 30))
        nb, ne = int(_log(rng, 1, 15)), rng.randint(1, 6)
        nx, ny = int(_log(rng, 32, side_max)), int(_log(rng, 32, side_max))
        n_psf = rng.randint(3, 6)
        if ns * n_psf * N_RADII * nb * ne * nx * ny <= PAIRS_MAX / 4:
            break
    if order == "store":  # a store's patches are whole super-pixels
        nx, ny = 8 * max(nx // 8, 4), 8 * max(ny // 8, 4)
    return dict(kind=kind, n_sources=ns, n_bands=nb, n_exp=ne, nx=nx, ny=ny, n_psf=n_psf,
                order=order)


# ------------------------------------------------------------------ inputs
def _spec(case):
    ns, nb = case["n_sources"], case["n_bands"]
    common = dict(n_psf=case["n_psf"], psf_sigma=(0.5, 4.0), rot_deg=1.0, scale_frac=0.02,
                  g_range=(0.8, 1.2), mask_frac=0.02, flux_sigma=1.0 if ns == 1 else 1.5,
                  position="centre" if ns == 1 else "uniform")
    if ns > 30:  # crowded fields hold bright, extended galaxies as well
        common.update(flux_sigma=3.0, bright_fraction=0.5)
    return synth.PatchSpec(n_sources=ns, exposures_per_band=[case["n_exp"]] * nb,
                           shapes=[(case["nx"], case["ny"])] * (nb * case["n_exp"]), **common)


def _store_order(P):
    """The pixels of every exposure in a pixel store's order: super-pixels by
    (x, y), y fastest inside each (all super-pixels whole)."""
    for e in range(len(P.exposure_N)):
        sl = slice(int(P.exposure_start[e]), int(P.exposure_start[e]) + int(P.exposure_N[e]))
        x, y = P.xpix[sl].astype(np.int64), P.ypix[sl].astype(np.int64)
        o = np.lexsort((y % 8, x % 8, y // 8, x // 8))
        for a in (P.xpix, P.ypix, P.data, P.ierr):
            a[sl] = a[sl][o]


def _patch(case, seed, return_residual=False):
    P = synth.make_patch(_spec(case), seed=seed, render=_render64,
                         return_residual=return_residual)
    if case.get("order") == "store":
        _store_order(P)
    return P


def _uneven_patches(case, seed):
    rng = np.random.default_rng(case["layout"])   # the patches' sizes; the seed draws the rest
    seeds = np.random.default_rng(seed).integers(2 ** 31, size=case["n_patches"])
    out = []
    for s in seeds:
        nb = int(rng.integers(1, case["max_bands"] + 1))
        epb = [int(rng.integers(1, case["max_exp"] + 1)) for _ in range(nb)]
        sides = np.round(rng.uniform(32, case["max_side"], size=sum(epb))).astype(int)
        spec = synth.PatchSpec(n_sources=int(rng.integers(1, case["max_sources"] + 1)),
                               exposures_per_band=epb, shapes=[(int(w), int(w)) for w in sides],
                               n_psf=case["n_psf"], psf_sigma=(0.5, 4.0), rot_deg=1.0,
                               scale_frac=0.02, g_range=(0.8, 1.2), mask_frac=0.02,
                               flux_sigma=1.5)
        out.append(synth.make_patch(spec, seed=int(s), render=_render64))
    return out


def _chain_params(P, n_chains, seed):
    rng = np.random.default_rng(seed + 1)
    return P.truth[None] * (1.0 + 0.01 * rng.standard_normal((n_chains,) + P.truth.shape))


def _store_inputs(case, seed):
    """Exposures (float32, CUDA), regions (one list of records per patch) and
    background levels of a store call."""
    rng = np.random.default_rng(case["layout"])   # pointings and regions
    gen = torch.Generator(device="cuda").manual_seed(seed)
    side, n_exp, ns = case["side"], case["n_exp"], case["side"] // 8
    exps = []
    for _ in range(n_exp):
        e = torch.randn((ns, ns, 128), generator=gen, dtype=torch.float32, device="cuda")
        flux, ierr = e[..., :64], e[..., 64:]
        flux.mul_(0.05)
        flux[ierr > 3.0] = 20.0            # a few bright pixels
        ierr.copy_(torch.where(ierr < -2.0, 0.0, 20.0))   # and masked ones
        exps.append(e)
    ra0, dec0 = 53.16, synth.DEC0
    deg = synth.PIXEL_SCALE / 3600.0
    cosd = math.cos(math.radians(dec0))
    wcses = []
    for _ in range(n_exp):
        sh = rng.uniform(-0.02, 0.02, 2) * side * deg
        wcses.append(TanWCS(synth.store_header("F200W", (side, side),
                                               (ra0 + sh[0] / cosd, dec0 + sh[1]),
                                               (side / 2.0, side / 2.0), rng.uniform(-20, 20))))
    recs = np.zeros((case["n_patches"], n_exp), dtype=REGION_DTYPE)
    for p in range(case["n_patches"]):
        off = rng.uniform(-0.3, 0.3, 2) * side * deg
        ra, dec, rad = ra0 + off[0] / cosd, dec0 + off[1], case["radius"] * deg
        for i, w in enumerate(wcses):
            if case["shape"] == "circle":
                x, y = w.world_to_pixel_values(ra, dec)
                kind, par = REGION_CIRCLE, [float(x), float(y), case["radius"] ** 2]
            else:
                kind, par = RectangularRegion(ra - rad / cosd, ra + rad / cosd, dec - rad,
                                              dec + rad).device_params(w)
            recs[p, i]["kind"] = kind
            recs[p, i]["p"][:len(par)] = par
    bg = np.random.default_rng(seed).normal(0.0, 0.01, size=recs.shape).astype(np.float32)
    return exps, recs.reshape(-1), bg.reshape(-1) if case["background"] else None


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pack":
        exps, recs, bg = _store_inputs(case, seed)
        store = DeviceStore(case["side"], super_pixel_size=8, max_exposures=len(exps))
        for e in exps:
            store.add(e)
        idx = np.tile(np.arange(len(exps), dtype=np.int32), case["n_patches"])
        return dict(kind=kind, store=store, idx=idx, recs=recs, bg=bg, max_snr=case["max_snr"])
    if kind == "batch":
        patches = _uneven_patches(case, seed)
        for P in patches:
            P.send_to_device()
        batch = PatchBatch(patches)
        dprop, chi2, dchi2 = batch.device_buffers()
        return dict(kind=kind, patches=patches, batch=batch, dprop=dprop, chi2=chi2, dchi2=dchi2)
    P = _patch(case, seed, return_residual=kind == "residual")
    if kind == "chains":
        nch, ns, nb = case["n_chains"], case["n_sources"], case["n_bands"]
        copies = [ChainCopy(P) for _ in range(nch)]
        batch = PatchBatch(copies)
        theta = torch.as_tensor(_chain_params(P, nch, seed).reshape(-1), **F64)
        return dict(kind=kind, patch=P, copies=copies, batch=batch, theta=theta,
                    table=DeviceSersicTable(P.table),
                    src_bands=torch.full((nch * ns,), nb, dtype=torch.int32, device="cuda"),
                    src_off=torch.arange(nch * ns, dtype=torch.int64, device="cuda") * (nb + 6),
                    dprop=torch.zeros(nch * ns * SOURCE_BYTES, dtype=torch.uint8, device="cuda"),
                    chi2=torch.zeros(batch.n_bands_total, **F64),
                    dchi2=torch.zeros(batch.n_dchi2, dtype=torch.float32, device="cuda"))
    P.send_to_device()
    state = dict(kind=kind, patch=P)
    if kind in ("evaluate", "residual"):
        state.update(proposer=GPUProposer(), prop=P.proposal())
    elif kind == "forward":
        state["theta"] = torch.as_tensor(P.params, **F64)
        state["ev"] = PatchEvaluator(P, mode="recompute")
    elif kind == "autograd":
        state["theta"] = torch.tensor(P.params, dtype=torch.float32, device="cuda",
                                      requires_grad=True)
        state["ev"] = PatchEvaluator(P)
    elif kind == "flux":
        state["scene"] = P.set_scene(np.arange(case["n_sources"]))
    return state


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "evaluate":
        chi2, dchi2 = state["proposer"].evaluate_proposal(state["prop"], patch=state["patch"])
        return dict(chi2=chi2, dchi2=dchi2)
    if kind == "residual":
        chi2, dchi2, res = state["proposer"].evaluate_proposal(
            state["prop"], patch=state["patch"], unpack=False)
        return dict(chi2=chi2, dchi2=dchi2, residual=res)
    if kind == "forward":
        state["ev"].run(state["theta"], grad=False)
        return dict(chi2=state["ev"].chi2)
    if kind == "autograd":
        theta = state["theta"]
        theta.grad = None
        lnp = lnlike(theta.double(), state["ev"])
        lnp.backward()
        return dict(lnp=lnp.detach(), grad=theta.grad)
    if kind == "batch":
        state["batch"].evaluate_device(state["dprop"], state["chi2"], state["dchi2"])
        return dict(chi2=state["chi2"], dchi2=state["dchi2"])
    if kind == "chains":
        state["table"].build_proposal_batch(state["theta"], state["src_bands"],
                                            state["src_off"], state["dprop"])
        state["batch"].evaluate_device(state["dprop"], state["chi2"], state["dchi2"])
        return dict(chi2=state["chi2"], dchi2=state["dchi2"])
    if kind == "flux":
        flux, precision = optimize_fluxes_device(state["patch"], state["scene"])
        return dict(flux=flux, precision=precision)
    (data, ierr, x, y), start, n = state["store"].gather(
        state["idx"], state["recs"], background=state["bg"], max_snr=state["max_snr"])
    return dict(data=data, ierr=ierr, x=x, y=y, start=start, n=n)


# ------------------------------------------------------------------ the least work
def _patch_work(ns, nb, n_exp_total, npix_exp, n_psf, grad, residual):
    """Pixels are read once (16 bytes).  A (pixel, Gaussian) pair counts where
    the Gaussian's exp-argument can stay below the cutoff: ellipses of 6 sigma
    for the mixture radii (0.01 to 1 arcsec, spread in their logarithm) over a
    PSF of 0.5 to 4 pixels, cut at the patch.  20 operations a pair for the
    model, 30 more for the gradient."""
    side2 = float(npix_exp)
    reach = 0.0
    for k in range(N_RADII):
        r = 0.01 * 100.0 ** (k / (N_RADII - 1.0)) / synth.PIXEL_SCALE
        for sig in (0.5 + 3.5 * (j + 0.5) / 4 for j in range(4)):
            area = math.pi * CUTOFF * (0.5 * r * r + sig * sig)
            reach += 0.6 * min(1.0, area / side2) / (4 * N_RADII)
    pairs = reach * ns * n_psf * N_RADII * n_exp_total * npix_exp
    nbytes = n_exp_total * npix_exp * (20 if residual else 16) + ns * SOURCE_BYTES + 8 * nb
    nbytes += 28 * ns * nb if grad else 0
    return dict(bytes=float(nbytes), flops=pairs * (50.0 if grad else 20.0))


def work(case):
    kind = case["kind"]
    if kind == "pack":
        area = math.pi * case["radius"] ** 2 if case["shape"] == "circle" \
            else 4 * case["radius"] ** 2
        pix = case["n_patches"] * case["n_exp"] * area
        return dict(bytes=24.0 * pix, flops=4.0 * pix)
    if kind == "batch":
        one = _patch_work((1 + case["max_sources"]) / 2, (1 + case["max_bands"]) / 2,
                          (1 + case["max_bands"]) * (1 + case["max_exp"]) / 4,
                          (32 ** 2 + 32 * case["max_side"] + case["max_side"] ** 2) / 3,
                          case["n_psf"], True, False)
        return {k: v * case["n_patches"] for k, v in one.items()}
    npix_exp = 64 * (-(-case["nx"] // 8)) * (-(-case["ny"] // 8))
    ns, nb = case["n_sources"], case["n_bands"]
    w = _patch_work(ns, nb, nb * case["n_exp"], npix_exp, case["n_psf"],
                    kind not in ("forward", "flux"), kind == "residual")
    if kind == "chains":
        w = {k: v * case["n_chains"] for k, v in w.items()}
    if kind == "flux":  # unit-flux models, then products of all pairs of sources
        w["flops"] += float(ns * (ns + 3)) * nb * case["n_exp"] * npix_exp
        w["bytes"] += 8.0 * nb * ns * (ns + 1)
    return w


# ------------------------------------------------------------------ 64 bits
def _sources64(prop):
    """Leaves of one proposal's parameters in 64 bits; the amplitudes are
    linear in the last two about the proposal."""
    t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), **F64)
    src = {k: t(prop[k]).requires_grad_(True) for k in ("ra", "dec", "q", "pa")}
    src["flux"] = t(prop["fluxes"]).requires_grad_(True)
    src["dn"] = torch.zeros(len(prop), **F64).requires_grad_(True)
    src["drh"] = torch.zeros(len(prop), **F64).requires_grad_(True)
    src["amps"] = t(prop["mixture_amplitudes"]) \
        + src["dn"][:, None] * t(prop["damplitude_dnsersic"]) \
        + src["drh"][:, None] * t(prop["damplitude_drh"])
    return src


def _gaussians64(P, src, band, e):
    """(A, x, y, Fxx, Fyy, Fxy) of exposure e's image Gaussians, (n_sources * n_psf,)."""
    t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), **F64)
    p0, npsf = int(P.psfgauss_start[e]), int(P.n_psf_per_source[band])
    psf = P.psfgauss[p0:p0 + npsf]
    k = torch.as_tensor(psf["sersic_bin"].astype(np.int64), device="cuda")
    D, CW = t(P.D[e]), t(P.CW[e])
    c, s = torch.cos(src["pa"]), torch.sin(src["pa"])
    q = src["q"]
    R = torch.stack([torch.stack([c, -s], -1), torch.stack([s, c], -1)], -2)
    T = D @ R @ torch.diag_embed(torch.stack([1.0 / q, q], -1))
    TT = T @ T.transpose(-1, -2)
    r2 = t(P.rad2)[k]
    Sxx = TT[:, 0, 0, None] * r2 + t(psf["Cxx"])
    Syy = TT[:, 1, 1, None] * r2 + t(psf["Cyy"])
    Sxy = TT[:, 0, 1, None] * r2 + t(psf["Cxy"])
    det = Sxx * Syy - Sxy * Sxy
    d = torch.stack([src["ra"], src["dec"]], -1) - t(P.crval[e])
    cen = (CW @ d[..., None])[..., 0] + t(P.crpix[e])
    A = float(P.G[e]) * t(psf["amp"]) / torch.sqrt(det) / (2 * math.pi) \
        * src["flux"][:, band, None] * src["amps"][:, k]
    out = (A, cen[:, 0, None] + t(psf["xcen"]), cen[:, 1, None] + t(psf["ycen"]), Syy / det,
           Sxx / det, -Sxy / det)
    return [v.expand(A.shape).reshape(-1) for v in out]


def _shape64(g, x, y):
    """G H of every Gaussian at pixels (x, y), and what its derivatives need."""
    _, xc, yc, fxx, fyy, fxy = (v.detach()[:, None] for v in g)
    dx, dy = x[None] - xc, y[None] - yc
    vx, vy = fxx * dx + fxy * dy, fyy * dy + fxy * dx
    Q = dx * vx + dy * vy
    G = torch.where(Q > CUTOFF, 0.0, torch.exp(-0.5 * Q))
    H = 1.0 + (vx * vx + vy * vy - fxx - fyy) / 24.0
    return dx, dy, vx, vy, G, H


def _chunks(n, n_gauss):
    step = max(64, int(2e7 / max(n_gauss, 1)))
    return [slice(i, min(i + step, n)) for i in range(0, n, step)]


def _pixels64(P, e):
    p0, n = int(P.exposure_start[e]), int(P.exposure_N[e])
    return p0, n, [torch.as_tensor(a[p0:p0 + n].astype(np.float64), **F64)
                   for a in (P.xpix, P.ypix, P.data, P.ierr)]


def _exposures(P):
    for b in range(len(P.band_start)):
        for e in range(int(P.band_start[b]), int(P.band_start[b]) + int(P.band_N[b])):
            yield b, e


def _render64(P, params):
    src = _sources64(proposal_from_params(params, P.n_bands, P.table))
    model = np.zeros(P.npix)
    with torch.no_grad():
        for b, e in _exposures(P):
            g = _gaussians64(P, src, b, e)
            p0, n, (x, y, _, _) = _pixels64(P, e)
            out = torch.empty(n, **F64)
            for sl in _chunks(n, len(g[0])):
                *_, G, H = _shape64(g, x[sl], y[sl])
                out[sl] = g[0] @ (G * H)
            model[p0:p0 + n] = out.cpu().numpy()
    return model


def _evaluate64(P, prop, grad=True):
    """chi2 (n_bands,), dchi2 (n_bands, n_sources, 7), residual (npix,)."""
    nb, ns = P.n_bands, len(prop)
    chi2, res = np.zeros(nb), np.zeros(P.npix)
    dchi2 = np.zeros((nb, ns, 7))
    src = _sources64(prop)
    leaves = [src[k] for k in ("flux", "ra", "dec", "q", "pa", "dn", "drh")]
    for b, e in _exposures(P):
        g = _gaussians64(P, src, b, e)
        A, _, _, fxx, fyy, fxy = (v.detach() for v in g)
        p0, n, (x, y, data, ierr) = _pixels64(P, e)
        sums = torch.zeros((6, len(A)), **F64)
        r = torch.empty(n, **F64)
        for sl in _chunks(n, len(A)):
            dx, dy, vx, vy, G, H = _shape64(g, x[sl], y[sl])
            r[sl] = data[sl] - A @ (G * H)
            if not grad:
                continue
            W = (-2.0 * r[sl] * ierr[sl] ** 2)[None] * G
            WH = W * H
            Vx, Vy, S = (W * vx).sum(1), (W * vy).sum(1), W.sum(1)
            sums[0] += WH.sum(1)
            sums[1] += A * ((WH * vx).sum(1) - (fxx * Vx + fxy * Vy) / 12.0)
            sums[2] += A * ((WH * vy).sum(1) - (fxy * Vx + fyy * Vy) / 12.0)
            sums[3] += A * ((W * dx * vx).sum(1) / 12.0 - 0.5 * (WH * dx * dx).sum(1) - S / 24.0)
            sums[4] += A * ((W * dy * vy).sum(1) / 12.0 - 0.5 * (WH * dy * dy).sum(1) - S / 24.0)
            sums[5] += A * ((W * (dx * vy + dy * vx)).sum(1) / 12.0 - (WH * dx * dy).sum(1))
        chi2[b] += float((ierr ** 2 * (r * r - data * data)).sum())
        res[p0:p0 + n] = r.cpu().numpy()
        if grad:
            gs = torch.autograd.grad(g, leaves, grad_outputs=list(sums), retain_graph=True)
            cols = [gs[0][:, b]] + list(gs[1:])
            dchi2[b] += torch.stack(cols, -1).cpu().numpy()
    return chi2, dchi2, res


def _basis64(t, x):
    """The four cubic B-splines on knots t that are not zero at x (clamped to
    the knots' range), their derivatives, and the first one's index."""
    x = min(max(x, t[3]), t[-4])
    i = min(max(int(np.searchsorted(t, x, side="right")) - 1, 3), len(t) - 5)

    def spline(j, k):
        if k == 0:
            return 1.0 if j == i else 0.0
        a, b = t[j + k] - t[j], t[j + k + 1] - t[j + 1]
        return ((x - t[j]) / a * spline(j, k - 1) if a else 0.0) + \
            ((t[j + k + 1] - x) / b * spline(j + 1, k - 1) if b else 0.0)

    def slope(j):
        a, b = t[j + 3] - t[j], t[j + 4] - t[j + 1]
        return 3.0 * ((spline(j, 2) / a if a else 0.0) - (spline(j + 1, 2) / b if b else 0.0))

    js = range(i - 3, i + 1)
    return i - 3, np.array([spline(j, 3) for j in js]), np.array([slope(j) for j in js])


def _proposal64(params, nb, table):
    """Proposal fields in 64 bits (a dict) of parameters (n_sources, n_bands + 6)."""
    tx, ty, c = table.knots_and_coeffs()
    p = np.asarray(params, dtype=np.float64)
    prop = np.zeros(len(p), dtype=[(k, "f8") for k in ("ra", "dec", "q", "pa")] +
                    [("fluxes", "f8", nb)] +
                    [(k, "f8", N_RADII) for k in ("mixture_amplitudes", "damplitude_dnsersic",
                                                  "damplitude_drh")])
    prop["fluxes"] = p[:, :nb]
    for k, name in enumerate(("ra", "dec", "q", "pa")):
        prop[name] = p[:, nb + k]
    for s, (nser, rh) in enumerate(p[:, nb + 4:nb + 6]):
        i, bx, dbx = _basis64(tx, nser)
        j, by, dby = _basis64(ty, rh)
        w = c[:, i:i + 4, j:j + 4]
        for name, u, v in (("mixture_amplitudes", bx, by), ("damplitude_dnsersic", dbx, by),
                           ("damplitude_drh", bx, dby)):
            prop[name][s] = np.einsum("kab,a,b->k", w, u, v)
    return prop


def _fluxes64(P, prop):
    """Fluxes (n_bands, n_sources) and precisions of the weighted least squares."""
    nb, ns = P.n_bands, len(prop)
    flux, ata = torch.zeros((nb, ns), **F64), torch.zeros((nb, ns, ns), **F64)
    unit = prop.copy()
    unit["fluxes"] = 1.0
    src = _sources64(unit)
    atb = torch.zeros((nb, ns), **F64)
    with torch.no_grad():
        for b, e in _exposures(P):
            g = _gaussians64(P, src, b, e)
            _, n, (x, y, data, ierr) = _pixels64(P, e)
            for sl in _chunks(n, len(g[0])):
                *_, G, H = _shape64(g, x[sl], y[sl])
                X = (g[0][:, None] * G * H).view(ns, -1, G.shape[1]).sum(1) * ierr[sl]
                ata[b] += X @ X.T
                atb[b] += X @ (data[sl] * ierr[sl])
        flux = torch.linalg.solve(ata, atb[..., None])[..., 0]
    return flux, ata


def _pack64(case, seed):
    exps, recs, bg = _store_inputs(case, seed)
    n_exp, ns = len(exps), case["side"] // 8
    lo = torch.arange(ns, **F64) * 8.0
    k = torch.arange(64, device="cuda")
    out, n = [[], [], [], []], []
    for i, rec in enumerate(recs):
        xc, yc, r2 = (float(v) for v in rec["p"][:3])
        dx = torch.minimum((xc - lo) ** 2, (xc - lo - 7.0) ** 2)
        dy = torch.minimum((yc - lo) ** 2, (yc - lo - 7.0) ** 2)
        sx, sy = torch.nonzero(dx[:, None] + dy[None] < r2, as_tuple=True)
        sp = exps[i % n_exp][sx, sy].to(torch.float64)
        flux, ierr = sp[:, :64], sp[:, 64:]
        if bg is not None:
            flux = flux - float(bg[i])
        if case["max_snr"] > 0:
            ierr = torch.where((ierr > 0) & (flux * ierr > case["max_snr"]),
                               case["max_snr"] / flux, ierr)
        for o, v in zip(out, (flux, ierr, sx[:, None] * 8.0 + k // 8, sy[:, None] * 8.0 + k % 8)):
            o.append(v.reshape(-1).to(torch.float64))
        n.append(64 * len(sx))
    data, ierr, x, y = (torch.cat(o) for o in out)
    n = np.array(n, dtype=np.int32)
    start = np.concatenate([[0], np.cumsum(n)[:-1]]).astype(np.int32)
    return dict(data=data, ierr=ierr, x=x, y=y, start=start, n=n)


def exact(case, seed):
    kind = case["kind"]
    if kind == "pack":
        # a box's edge test goes through the sky projection: no value in its place
        return _pack64(case, seed) if case["shape"] == "circle" else None
    if kind == "batch":
        got = [_evaluate64(P, P.proposal()) for P in _uneven_patches(case, seed)]
        return dict(chi2=np.concatenate([c for c, _, _ in got]),
                    dchi2=np.concatenate([d.reshape(-1) for _, d, _ in got]))
    P = _patch(case, seed)
    nb = P.n_bands
    if kind in ("evaluate", "residual"):
        chi2, dchi2, res = _evaluate64(P, P.proposal())
        out = dict(chi2=chi2, dchi2=dchi2)
        return dict(out, residual=res) if kind == "residual" else out
    if kind == "forward":
        return dict(chi2=_evaluate64(P, _proposal64(P.params, nb, default_table()), False)[0])
    if kind == "autograd":
        theta = P.params.astype(np.float32).astype(np.float64)
        chi2, d, _ = _evaluate64(P, _proposal64(theta, nb, default_table()))
        grad = np.concatenate([d[:, :, 0].T, d[:, :, 1:].sum(0)], axis=1)
        return dict(lnp=-0.5 * chi2.sum(), grad=-0.5 * grad)
    if kind == "chains":
        got = [_evaluate64(P, _proposal64(th, nb, default_table()))
               for th in _chain_params(P, case["n_chains"], seed)]
        return dict(chi2=np.concatenate([c for c, _, _ in got]),
                    dchi2=np.concatenate([d.reshape(-1) for _, d, _ in got]))
    flux, ata = _fluxes64(P, P.proposal())
    return dict(flux=flux, precision=ata)
