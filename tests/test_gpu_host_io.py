"""GPU: what host pointers may be in an evaluation with host buffers and in the
retrieval of a pixel array: pageable and pinned memory, and pinned memory that
earlier work in the stream still has to fill."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def case(ns):
    from forcepho_b200 import synth
    P = synth.make_patch(synth.PatchSpec(n_sources=ns, exposures_per_band=[1],
                                         shapes=[(32, 32)], n_psf=2), seed=5)
    P.return_residual = True
    P.send_to_device()
    return P, P.proposal()


def evaluate(P, ptr, flags):
    from forcepho_b200 import _lib
    import torch
    ns = P.n_sources
    chi2, dchi2 = np.zeros(P.n_bands), np.zeros((P.n_bands, 7 * ns), np.float32)
    _lib.call("fpho_evaluate_proposal", P.device_patch.handle, ptr, ns, chi2.ctypes.data,
              dchi2.ctypes.data, 7 * ns, flags, torch.cuda.current_stream().cuda_stream)
    return chi2, dchi2


@pytest.mark.parametrize("ns", [1, 4, 5, 15, 16, 64, 65])
def test_proposal_memory(ns):
    """Sizes either side of each form of the first launch."""
    import torch
    from forcepho_b200 import _lib
    P, prop = case(ns)
    raw = np.frombuffer(prop.tobytes(), dtype=np.uint8).copy()
    want = evaluate(P, raw.ctypes.data, _lib.FPHO_IO_HOST)
    assert want[0].all()
    dev = torch.from_numpy(raw).cuda()
    pinned = torch.zeros(len(raw), dtype=torch.uint8).pin_memory()
    a = torch.rand(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    for _ in range(8):                      # some milliseconds ahead of the copy
        a = a @ a * 1e-4
    pinned.copy_(dev, non_blocking=True)
    for _ in range(2):                      # not filled yet; then filled
        got = evaluate(P, pinned.data_ptr(), _lib.FPHO_IO_HOST)
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)
    P.free()


def test_retrieve_memory():
    import torch
    from forcepho_b200 import _lib
    P, _ = case(1)
    n = len(P.data)
    out, pinned = np.zeros(n, np.float32), torch.zeros(n).pin_memory()

    def retrieve(ptr):
        _lib.call("fpho_patch_retrieve", P.device_patch.handle, 0, ptr, None)

    retrieve(out.ctypes.data)
    retrieve(pinned.data_ptr())
    np.testing.assert_array_equal(out, P.data)
    np.testing.assert_array_equal(pinned.numpy(), P.data)
    P.free()
