"""GPU parity over the ways in which a patch's tiles are run -- one, two or four
CTAs a tile, persistent CTAs over many tiles, tiles of several patches -- each in
the pixel orders that the kernels tell apart.  Bars: those of test_gpu_parity."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import CHI2_RTOL, check_grad
from test_gpu_runs import patch, reorder

pytestmark = pytest.mark.gpu

ORDERS = ["morton", "store", "shuffled"]


def tile_form(P):
    """(persistent, CTAs per tile) of the next evaluation."""
    from forcepho_b200 import _lib
    out = (ctypes.c_int * 2)()
    _lib.call("fpho_patch_tile_form", P.device_patch.handle, out)
    return tuple(out)


def check(P, prop, variant=None, form=None):
    from forcepho_b200.proposal import GPUProposer
    for residual in (False, True):
        P.return_residual = residual
        P.free()
        P.send_to_device()
        if variant is not None:
            P.device_patch.set_config(variant, 256)
        if form is not None:
            assert tile_form(P) == form
        c, g, r = O.oracle_evaluate(P, prop, residual=True)
        for _ in range(2):          # (the second in the order of the first's costs)
            chi2, dchi2, *res = GPUProposer().evaluate_proposal(prop, patch=P, unpack=False)
            np.testing.assert_allclose(chi2, c, rtol=CHI2_RTOL)
            check_grad(dchi2, g, P, prop)
            if residual:
                assert np.max(np.abs(res[0] - r)) <= 1e-5 * np.abs(P.data).max()
    P.free()


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("n_exp,form", [(2, (0, 4)), (4, (0, 2)), (9, (0, 1)), (27, (0, 1)),
                                        (40, (1, 1))])
def test_forms(n_exp, form, order):
    """32, 64, 144, 432 and 640 tiles of 256 pixels."""
    if sms() != 148:
        pytest.skip("the forms of these sizes are those of 148 SMs")
    P = reorder(patch(2, [n_exp // 2, n_exp - n_exp // 2], [(64, 64)] * n_exp, 2, seed=61), order)
    check(P, P.proposal(), form=form)


@pytest.mark.parametrize("order", ["morton", "store", "rows16", "columns", "shuffled"])
@pytest.mark.parametrize("variant", [9, 10, 12])
def test_unparted_split(variant, order):
    """The split form with a whole tile per CTA, 2, 4 and 8 warps."""
    P = reorder(patch(4, [2, 1], [(48, 32), (32, 32), (64, 48)], 4, seed=31), order)
    P.ierr[:24] = 0.0                 # whole runs without weight
    check(P, P.proposal(), variant, (0, 1))


@pytest.mark.parametrize("variant", [None, 8])
@pytest.mark.parametrize("order", ORDERS)
def test_batches(order, variant):
    from forcepho_b200.batch import PatchBatch
    patches = [reorder(patch(ns, [ne], [(48, 40)] * ne, 3, seed=70 + ns), order)
               for ns, ne in ((1, 1), (5, 3), (3, 2))]
    for P in patches:
        P.return_residual = False
        P.send_to_device()
    batch = PatchBatch(patches) if variant is None else PatchBatch(patches, variant=variant)
    props = [P.proposal() for P in patches]
    for P, q, chi2, dchi2 in zip(patches, props, *batch.evaluate(props)):
        c, g = O.oracle_evaluate(P, q)
        np.testing.assert_allclose(chi2, c, rtol=CHI2_RTOL)
        check_grad(np.asarray(dchi2).reshape(g.shape), g, P, q)
    batch.free()
    for P in patches:
        P.free()
