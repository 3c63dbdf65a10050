"""GPU: patches whose kernels need all but the last few hundred bytes of an SM's
shared memory (227 KB a CTA, 128 bytes of it static)."""
import numpy as np
import pytest

from test_gpu_runs import patch

pytestmark = pytest.mark.gpu

LIMIT = 227 * 1024 - 128


def tight(ns, n_psf):
    """One small exposure under many sources."""
    P = patch(ns, [1], [(16, 16)], n_psf, seed=91)
    P.return_residual = False
    P.send_to_device()
    return P


@pytest.mark.parametrize("variant,live_cap,ns,n_psf", [
    (4, 32, 771, 2), (4, 48, 764, 2), (2, 32, 771, 2), (10, 32, 743, 2)])
def test_tile_kernel_at_the_limit(variant, live_cap, ns, n_psf):
    """The sizes 8 warps x (7 floats a source) + a word a Gaussian + 128 bytes a
    staged record (+ the split form's partial models) leave no room for more."""
    from forcepho_b200.proposal import GPUProposer
    need = 128 * live_cap + ns * (8 * 28 + 4 * 9 * n_psf) + (8 * 256 * 4 if variant == 10 else 0)
    assert LIMIT - 512 < need <= LIMIT
    P = tight(ns, n_psf)
    prop = P.proposal()
    chi2, dchi2 = GPUProposer().evaluate_proposal(prop, patch=P, unpack=False)
    P.device_patch.set_config(variant, live_cap)
    c, g = GPUProposer().evaluate_proposal(prop, patch=P, unpack=False)
    np.testing.assert_allclose(c, chi2, rtol=1e-6)
    # 700 sources on 256 pixels: the residual's rounding is what the forms share
    assert np.linalg.norm(g - dchi2) <= 1e-3 * np.linalg.norm(dchi2)
    P.free()


def test_normal_equations_at_the_limit():
    import torch
    from forcepho_b200 import _lib
    ns, n_psf = 160, 10
    assert LIMIT - 512 < 64 * 128 + 2 * 256 * 4 + ns * (257 * 4 + 4 * 9 * n_psf) <= LIMIT
    P = tight(ns, n_psf)
    prop = torch.from_numpy(np.frombuffer(P.proposal().tobytes(), dtype=np.uint8).copy()).cuda()
    ata = torch.zeros(ns, ns, dtype=torch.float64, device="cuda")
    atb = torch.zeros(ns, dtype=torch.float64, device="cuda")
    _lib.call("fpho_patch_flux_normal_equations", P.device_patch.handle, prop.data_ptr(), ns,
              ata.data_ptr(), atb.data_ptr(), torch.cuda.current_stream().cuda_stream)
    X = P.design_matrix_device(P.proposal()).double() * torch.from_numpy(P.ierr).cuda().double()
    want = X @ X.T
    torch.testing.assert_close(ata, want, rtol=0, atol=1e-9 * float(want.abs().max()))
    P.free()
