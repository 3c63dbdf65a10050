"""GPU parity over the pixel orders the tile kernels tell apart: runs of eight
pixels that share y (x fastest inside a super-pixel), that share x (a pixel
store's order), runs of a longer super-pixel row, and pixels in no order at
all; with ragged exposures, padding and masked runs; and at the sizes where a
tile is dealt to one, two or four CTAs.

Bars: those of test_gpu_parity (chi2 1e-6 against the float oracle, gradients
per component by check_grad)."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import CHI2_RTOL, check_grad, gpu_eval

pytestmark = pytest.mark.gpu


def reorder(P, order, seed=0):
    """The pixels of every exposure of `P` in another packed order."""
    rng = np.random.default_rng(seed)
    for e in range(len(P.exposure_N)):
        sl = slice(int(P.exposure_start[e]), int(P.exposure_start[e]) + int(P.exposure_N[e]))
        x, y = P.xpix[sl].astype(np.int64), P.ypix[sl].astype(np.int64)
        if order == "store":          # super-pixels by (x, y), y fastest
            o = np.lexsort((y % 8, x % 8, y // 8, x // 8))
        elif order == "rows16":       # 16-pixel super-pixels, x fastest
            o = np.lexsort((x % 16, y % 16, x // 16, y // 16))
        elif order == "columns":      # whole columns
            o = np.lexsort((y, x))
        elif order == "shuffled":
            o = rng.permutation(len(x))
        else:
            o = np.arange(len(x))
        for a in (P.xpix, P.ypix, P.data, P.ierr):
            a[sl] = a[sl][o]
    return P


def patch(ns, exposures, shapes, npsf, seed, **kw):
    from forcepho_b200 import synth
    spec = synth.PatchSpec(n_sources=ns, exposures_per_band=exposures, shapes=shapes, n_psf=npsf,
                           psf_sigma=(0.5, 4.0), rot_deg=1.0, scale_frac=0.02, g_range=(0.8, 1.2),
                           mask_frac=0.05, flux_sigma=1.0, **kw)
    return synth.make_patch(spec, seed=seed)


@pytest.mark.parametrize("variant", [8, 6])
@pytest.mark.parametrize("order", ["morton", "store", "rows16", "columns", "shuffled"])
def test_pixel_orders(order, variant):
    P = reorder(patch(4, [2, 1], [(48, 32), (32, 32), (64, 48)], 4, seed=31), order)
    P.ierr[:24] = 0.0                 # whole runs without weight
    prop = P.proposal()
    for residual in (False, True):
        chi2, dchi2, *res = gpu_eval(P, prop, residual=residual, variant=variant, live_cap=256)
        c, g, r = O.oracle_evaluate(P, prop, residual=True)
        np.testing.assert_allclose(chi2, c, rtol=CHI2_RTOL)
        check_grad(dchi2, g, P, prop)
        if residual:
            assert np.max(np.abs(res[0] - r)) <= 1e-5 * np.abs(P.data).max()


@pytest.mark.parametrize("shapes", [[(17, 9)], [(97, 83)], [(40, 64)] * 7, [(128, 128)] * 3,
                                    [(128, 121)] * 5])
def test_tile_parts(shapes):
    """From one tile to a few per SM (one, two and four CTAs per tile), with
    padding in the odd shapes."""
    P = patch(2, [len(shapes)], shapes, 3, seed=33)
    prop = P.proposal()
    chi2, dchi2, res = gpu_eval(P, prop, residual=True)
    c, g, r = O.oracle_evaluate(P, prop, residual=True)
    np.testing.assert_allclose(chi2, c, rtol=CHI2_RTOL)
    check_grad(dchi2, g, P, prop)
    assert np.max(np.abs(res - r)) <= 1e-5 * np.abs(P.data).max()


@pytest.mark.parametrize("ns,nb", [(1, 1), (5, 3), (13, 8)])
def test_lnlike_gradient_forms(ns, nb):
    """The fused gradient of LnLike against the stacked torch form: plain,
    scaled by an upstream gradient, batched and under create_graph."""
    import torch
    from forcepho_b200.autograd import PatchEvaluator, lnlike
    P = patch(ns, [1] * nb, [(24, 24)] * nb, 2, seed=50 + ns)
    P.send_to_device()
    ev = PatchEvaluator(P)
    theta = torch.tensor(P.params, dtype=torch.float64, device="cuda", requires_grad=True)
    out = lnlike(theta, ev)
    assert float(out.detach()) == pytest.approx(-0.5 * float(ev.chi2.sum()), rel=1e-14)
    want = ev.stacked() * -0.5
    (g,) = torch.autograd.grad(out, theta, retain_graph=True)
    torch.testing.assert_close(g, want, rtol=1e-14, atol=0)
    (g3,) = torch.autograd.grad(3.0 * out, theta, retain_graph=True)
    torch.testing.assert_close(g3, 3.0 * want, rtol=1e-14, atol=0)
    seeds = torch.tensor([1.0, -2.0], dtype=torch.float64, device="cuda")
    (gb,) = torch.autograd.grad(out, theta, seeds, is_grads_batched=True, retain_graph=True)
    torch.testing.assert_close(gb, seeds[:, None, None] * want, rtol=1e-14, atol=0)
    w = torch.ones((), dtype=torch.float64, device="cuda", requires_grad=True)
    (gc,) = torch.autograd.grad(w * out, theta, create_graph=True)
    (dw,) = torch.autograd.grad(gc.sum(), w)
    torch.testing.assert_close(dw, want.sum(), rtol=1e-12, atol=0)
    P.free()


def test_lnlike_gradient_of_a_lazy_negative():
    """An upstream gradient whose sign is a flag on the tensor, not in memory."""
    import torch
    from forcepho_b200.autograd import PatchEvaluator, lnlike
    P = patch(2, [1], [(24, 24)], 2, seed=61)
    P.send_to_device()
    ev = PatchEvaluator(P)
    theta = torch.tensor(P.params, dtype=torch.float64, device="cuda", requires_grad=True)
    up = torch.tensor(1.0 + 2.0j, dtype=torch.complex128, device="cuda").conj().imag
    assert up.is_neg() and float(up) == -2.0
    (g,) = torch.autograd.grad(lnlike(theta, ev), theta, up)
    torch.testing.assert_close(g, ev.stacked(), rtol=1e-14, atol=0)
    P.free()
