"""The tile scan's kept lists against a restatement in double: long, thin
galaxies off the axes, of whose image Gaussians many reach a tile's box but not
the tile, so that every warp's queue for the exact test fills and empties
several times."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_runs import patch

pytestmark = pytest.mark.gpu


def min_exparg(box, g):
    """Smallest (p - c)^T F (p - c) over each box (x0, x1, y0, y1) for each
    image Gaussian (amp, xc, yc, fxx, fyy, fxy): (boxes, Gaussians), double."""
    x0, x1, y0, y1 = (box[:, k, None].astype(np.float64) for k in range(4))
    xc, yc, fxx, fyy, fxy = (g[None, :, k].astype(np.float64) for k in range(1, 6))
    best = np.full((len(box), len(g)), np.inf)
    for x in (x0, x1):
        dx = x - xc
        dy = np.clip(-fxy * dx / fyy, y0 - yc, y1 - yc)
        best = np.minimum(best, fxx * dx * dx + 2 * fxy * dx * dy + fyy * dy * dy)
    for y in (y0, y1):
        dy = y - yc
        dx = np.clip(-fxy * dy / fxx, x0 - xc, x1 - xc)
        best = np.minimum(best, fxx * dx * dx + 2 * fxy * dx * dy + fyy * dy * dy)
    inside = (xc >= x0) & (xc <= x1) & (yc >= y0) & (yc <= y1)
    return np.where(inside, 0.0, best)


def nearest_exparg(box, g):
    """The exp-argument at the point of each box nearest the centre."""
    xc, yc, fxx, fyy, fxy = (g[None, :, k].astype(np.float64) for k in range(1, 6))
    dx = np.clip(xc, box[:, 0, None], box[:, 1, None]) - xc
    dy = np.clip(yc, box[:, 2, None], box[:, 3, None]) - yc
    return fxx * dx * dx + 2 * fxy * dx * dy + fyy * dy * dy


def tile_boxes(P, e, tile):
    """Bounding boxes of the weighted pixels of exposure e's tiles, and counts."""
    s, n = int(P.exposure_start[e]), int(P.exposure_N[e])
    boxes, counts = [], []
    for t in range(s, s + n, tile):
        sl = slice(t, min(t + tile, s + n))
        w = P.ierr[sl] != 0
        x, y = P.xpix[sl][w], P.ypix[sl][w]
        boxes.append([x.min(), x.max(), y.min(), y.max()])
        counts.append(sl.stop - sl.start)
    return np.array(boxes, dtype=np.float64), np.array(counts)


def elongated(seed):
    P = patch(40, [1, 1], [(64, 64), (64, 48)], 5, seed=seed, rh=(0.2, 0.5))
    nb = P.n_bands
    rng = np.random.default_rng(seed)
    P.params[:, nb + 2] = rng.uniform(0.2, 0.3, P.n_sources)                    # q
    P.params[:, nb + 3] = rng.choice([-1, 1], P.n_sources) * rng.uniform(0.6, 1.0, P.n_sources)
    return P


def expected(P, prop, tile=256):
    """Pairs certainly kept, pairs possibly kept, and the largest number of
    Gaussians that one warp of four has to test exactly for one tile."""
    sure = maybe = asked = 0
    for b in range(P.n_bands):
        e = int(P.band_start[b])
        g = O.image_gaussians_f32(P, prop, b, e)
        box, count = tile_boxes(P, e, tile)
        q = min_exparg(box, g)
        sure += int((count[:, None] * (q <= 36.06)).sum())
        maybe += int((count[:, None] * (q <= 36.08)).sum())
        ask = (q <= 36.0) & (nearest_exparg(box, g) > 36.1)
        for w in range(4):
            mine = (np.arange(len(g)) // 32) % 4 == w
            asked = max(asked, int(ask[:, mine].sum(1).max()))
    return sure, maybe, asked


@pytest.mark.parametrize("seed", [1, 2])
@pytest.mark.parametrize("variant", [8, 9, 10])
def test_kept_lists_of_elongated_sources(seed, variant):
    from forcepho_b200 import _lib
    from forcepho_b200.proposal import GPUProposer
    P = elongated(seed)
    prop = P.proposal()
    sure, maybe, asked = expected(P, prop)
    assert asked > 32                 # kept Gaussians alone fill a warp's queue
    P.return_residual = False
    P.send_to_device()
    P.device_patch.set_config(variant, 256)
    _lib.call("fpho_patch_count_pairs", P.device_patch.handle, 1, None)
    for _ in range(3):
        GPUProposer().evaluate_proposal(prop, patch=P)
        n = ctypes.c_longlong()
        _lib.call("fpho_patch_count_pairs", P.device_patch.handle, 1, ctypes.byref(n))
        assert sure <= n.value <= maybe, (sure, n.value, maybe)
    P.free()
