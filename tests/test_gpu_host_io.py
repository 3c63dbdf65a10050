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


@pytest.mark.parametrize("name", ["rad2", "D", "crpix", "crval", "CW", "G"])
def test_pinned_metadata_in_stream_order(name):
    """Metadata in pinned memory that earlier work in the (non-blocking) stream
    still has to fill, when a patch is created and when its metadata are replaced."""
    import torch
    from forcepho_b200 import _lib
    from forcepho_b200.patches.device_patch import DevicePatch
    P, prop = case(3)
    raw = np.frombuffer(prop.tobytes(), dtype=np.uint8).copy()
    want = evaluate(P, raw.ctypes.data, _lib.FPHO_IO_HOST)
    good = getattr(P, name)
    dev = torch.from_numpy(good.copy()).cuda()
    pinned = torch.from_numpy(good * 1.5).pin_memory()
    setattr(P, name, pinned.numpy())
    s = torch.cuda.Stream()
    a = torch.rand(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    for replace in (False, True):
        pinned.mul_(1.5)
        with torch.cuda.stream(s):
            for _ in range(8):              # some milliseconds ahead of the copy
                a = a @ a * 1e-4
            pinned.copy_(dev, non_blocking=True)
            if replace:
                st = P.host_struct()
                _lib.call("fpho_patch_replace_meta", P.device_patch.handle, st.ctypes.data,
                          s.cuda_stream)
            else:
                P.device_patch.free()
                P.device_patch = DevicePatch(P, True, stream=s.cuda_stream)
            got = evaluate(P, raw.ctypes.data, _lib.FPHO_IO_HOST)
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


def test_retrieve_without_a_pinned_block():
    from forcepho_b200 import _lib
    P, _ = case(1)
    out = np.zeros(len(P.data), np.float32)
    _lib.call("fpho_test_fail_alloc", 1)
    try:
        _lib.call("fpho_patch_retrieve", P.device_patch.handle, 0, out.ctypes.data, None)
    finally:
        _lib.call("fpho_test_fail_alloc", 0)
    np.testing.assert_array_equal(out, P.data)
    P.free()
