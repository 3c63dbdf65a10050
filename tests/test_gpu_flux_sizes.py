"""GPU: the flux solve at the sizes where its kernels change shape -- one source
to the limits of the register solve (32), of the tensor-core normal equations
(63) and of the solve (64), ragged exposures, both pixel orders -- against
float64 numpy on the device design matrix (whose unit-flux rows are the same
floats), with the bars of test_gpu_fixed_design (relative 1e-9 of each band's
scale: both sides sum exact products in double)."""
import numpy as np
import pytest

from test_gpu_runs import patch, reorder

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["morton", "store", "shuffled"])
@pytest.mark.parametrize("ns", [1, 7, 8, 31, 32, 33, 63, 64])
def test_flux_solve_sizes(ns, order):
    import torch
    from forcepho_b200.fitting import optimize_fluxes, optimize_fluxes_device
    shapes = [(96, 80), (96, 80), (80, 96)] if order == "store" else [(97, 83), (96, 80), (90, 96)]
    P = reorder(patch(ns, [2, 1], shapes, 3, seed=40 + ns), order)
    P.send_to_device()
    scene = P.set_scene(np.arange(ns), params=P.truth)
    want_f, want_p = optimize_fluxes(P, scene)
    f, p, status = optimize_fluxes_device(P, scene, return_status=True)
    torch.cuda.synchronize()
    f, p, status = f.cpu().numpy(), p.cpu().numpy(), status.cpu().numpy()
    for b in range(P.n_bands):
        assert status[b] == 0
        np.testing.assert_allclose(p[b], want_p[b], rtol=0, atol=1e-9 * np.abs(want_p[b]).max())
        # the solution moves by its condition number times the rounding of ATA
        cond = np.linalg.cond(want_p[b])
        np.testing.assert_allclose(f[b], want_f[b], rtol=0,
                                   atol=max(1e-9, 1e-14 * cond) * np.abs(want_f[b]).max())
    P.free()
