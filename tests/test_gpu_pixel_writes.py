"""GPU: a caller that reaches the pixel arrays through the device struct may
write them in the stream and evaluate right after.  Every kernel that reads
pixels waits for the work before the evaluation's first kernel."""
import numpy as np
import pytest

from test_gpu_runs import patch

pytestmark = pytest.mark.gpu


def view(address, n, typestr):
    import torch

    class View:
        __cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "version": 3,
                                    "data": (address, False)}
    return torch.as_tensor(View(), device="cuda")


def device_array(P, name):
    """The patch's device array `name` as a torch tensor over its memory."""
    dt = P.patch_struct_dtype
    st = view(P.device_patch.device_struct, dt.itemsize, "|u1").cpu().numpy().view(dt)[0]
    return view(int(st[name]), int(P.npix), "<f4")


@pytest.mark.parametrize("n_exp", [1, 40])          # 16 tiles (in parts), 640 (persistent)
@pytest.mark.parametrize("variant", [0, 3, 8, 9])
def test_pixels_written_in_the_stream(variant, n_exp):
    import torch
    from forcepho_b200 import _lib
    P = patch(3, [n_exp], [(64, 64)] * n_exp, 2, seed=41)
    P.return_residual = False
    P.send_to_device()
    P.device_patch.set_config(variant, 256)
    prop = torch.from_numpy(np.frombuffer(P.proposal().tobytes(), dtype=np.uint8).copy()).cuda()
    ns, nb = P.n_sources, P.n_bands
    chi2 = torch.zeros(nb, dtype=torch.float64, device="cuda")
    dchi2 = torch.zeros(nb * 7 * ns, device="cuda")
    ata = torch.zeros(nb * ns * ns, dtype=torch.float64, device="cuda")
    atb = torch.zeros(nb * ns, dtype=torch.float64, device="cuda")
    data, ierr = device_array(P, "data"), device_array(P, "ierr")
    data0, ierr0 = data.clone(), ierr.clone()
    np.testing.assert_array_equal(data0.cpu().numpy(), P.data)
    a = torch.rand(2048, 2048, device="cuda")

    def run(flux):
        s = torch.cuda.current_stream().cuda_stream
        if flux:
            _lib.call("fpho_patch_flux_normal_equations", P.device_patch.handle, prop.data_ptr(),
                      ns, ata.data_ptr(), atb.data_ptr(), s)
            return [ata.clone(), atb.clone()]
        _lib.call("fpho_evaluate_proposal", P.device_patch.handle, prop.data_ptr(), ns,
                  chi2.data_ptr(), dchi2.data_ptr(), 7 * ns, 0, s)
        return [chi2.clone(), dchi2.clone()]

    for flux in (False, True):
        for k in (2.0, 3.0):
            for _ in range(3):
                a @ a
            data.copy_(data0 * k)
            ierr.copy_(ierr0 / k)
            got = run(flux)
            torch.cuda.synchronize()
            for g, w in zip(got, run(flux)):     # everything in place
                assert torch.isfinite(g).all() and torch.equal(g, w)
    P.free()
