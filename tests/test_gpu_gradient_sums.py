"""The gradient pass alone against double: sources so faint that every residual
is its datum, to the bit, so that the gradient's distance from the sum in double
over the same float Gaussians (the mixed oracle) is the rounding of the gradient
sums and of nothing else.  Long thin galaxies (q 0.2 to 0.4) over several pixels
and sub-pixel ones, where the terms of the exp-argument and of the derivatives
cancel, under data of one sign, where roundings that are alike do not average
out, and of both.

Bar, relative to the sum over pixels and Gaussians of |each term|: 1e-7 rms over the
components and 2^-20 for each.  A term carries some ten roundings of 2^-24, which
average out over the ten thousand and more terms of a component, and its sums a few more that do not."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import gpu_eval
from test_gpu_runs import patch, reorder

pytestmark = pytest.mark.gpu

RMS_BAR, MAX_BAR = 1e-7, 2.0 ** -20


def faint(seed, q, rh, one_sign, order, shape=(64, 64)):
    P = patch(6, [1, 1], [shape, shape], 4, seed=seed, rh=rh)
    nb = P.n_bands
    rng = np.random.default_rng(seed)
    P.params[:, nb + 2] = rng.uniform(*q, P.n_sources)
    P.params[:, nb + 3] = rng.uniform(-1.5, 1.5, P.n_sources)
    P.params[:, :nb] = 1e-10 * rng.uniform(0.5, 2.0, (P.n_sources, nb))
    d = 0.5 + np.abs(rng.standard_normal(P.npix))
    P.data[:] = d if one_sign else d * rng.choice([-1.0, 1.0], P.npix)
    P.ierr[:] = np.where(P.ierr != 0, rng.uniform(0.5, 1.5, P.npix), 0.0)
    return reorder(P, order, seed)


@pytest.mark.parametrize("variant", [8, 9, 3])
@pytest.mark.parametrize("order", ["morton", "store", "shuffled"])
@pytest.mark.parametrize("q,rh", [((0.2, 0.4), (0.2, 0.5)), ((0.2, 0.4), (0.03, 0.1)),
                                  ((0.4, 1.0), (0.05, 0.3))])
@pytest.mark.parametrize("one_sign", [True, False])
def test_gradient_sums(one_sign, q, rh, order, variant):
    P = faint(71, q, rh, one_sign, order)
    prop = P.proposal()
    _, want, _, scale, _ = O.oracle_mixed_abs(P, prop, terms=True)
    _, dchi2, res = gpu_eval(P, prop, residual=True, variant=variant, live_cap=256)
    np.testing.assert_array_equal(res[P.ierr != 0], P.data[P.ierr != 0])
    err = np.abs(dchi2 - want) / scale
    assert np.sqrt(np.mean(err ** 2)) <= RMS_BAR and err.max() <= MAX_BAR


@pytest.mark.parametrize("order", ["morton", "shuffled"])
def test_masked_pixels_far_away(order):
    """Coordinates of pixels without weight have no part in the gradient, however
    far off they are."""
    P = faint(72, (0.4, 1.0), (0.05, 0.3), True, order)
    P.ierr[:64] = 0.0                 # whole runs
    P.ierr[70:75] = 0.0               # and parts of one
    prop = P.proposal()
    _, want = gpu_eval(P, prop)[:2]
    far = P.ierr == 0
    P.xpix[far], P.ypix[far] = 1e12, -1e12
    _, dchi2 = gpu_eval(P, prop)[:2]
    assert np.all(np.isfinite(dchi2))
    np.testing.assert_allclose(dchi2, want, rtol=1e-4, atol=1e-6 * np.abs(want).max())
