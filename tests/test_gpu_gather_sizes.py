"""GPU: DeviceStore.gather over the shapes its kernels tell apart -- one and
several chunks per exposure, empty selections, super-pixel sides with a
compile-time and a run-time size and without vector copies, one and many
exposures -- against the selection and packing in numpy, bit for bit; and the
two halves of a gather."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pack_numpy(exps, idx, recs, s, bg, max_snr):
    out, n = [[], [], [], []], []
    k = np.arange(s * s)
    for i, rec in zip(idx, recs):
        a = exps[i]
        xc, yc, r2 = rec["p"][:3]
        lo_x, lo_y = np.arange(a.shape[0]) * float(s), np.arange(a.shape[1]) * float(s)
        dx = np.minimum((xc - lo_x) ** 2, (xc - (lo_x + s - 1)) ** 2)
        dy = np.minimum((yc - lo_y) ** 2, (yc - (lo_y + s - 1)) ** 2)
        sx, sy = np.nonzero(dx[:, None] + dy[None] < r2)
        d, e = a[sx, sy, :s * s].copy(), a[sx, sy, s * s:].copy()
        if bg is not None:
            d -= np.float32(bg[len(n)])
        if max_snr:
            m = (e > 0) & (d * e > np.float32(max_snr))
            e[m] = np.float32(max_snr) / d[m]
        for o, v in zip(out, (d, e, sx[:, None] * s + k // s, sy[:, None] * s + k % s)):
            o.append(v.reshape(-1).astype(np.float32))
        n.append(len(sx) * s * s)
    return [np.concatenate(o) for o in out], np.array(n)


def store(s, nside, n_exp, seed=0):
    from forcepho_b200.patches.device_store import DeviceStore
    rng = np.random.default_rng(seed)
    ns = nside // s
    exps = []
    st = DeviceStore(nside, super_pixel_size=s, max_exposures=n_exp)
    for _ in range(n_exp):
        a = rng.normal(0.0, 0.05, (ns, ns, 2 * s * s)).astype(np.float32)
        a[..., s * s:] = np.where(rng.uniform(size=(ns, ns, s * s)) < 0.05, 0.0, 20.0)
        a[rng.uniform(size=a.shape) < 0.002] = 15.0
        exps.append(a)
        st.add(a)
    return st, exps, rng


def circles(idx, nside, radii, rng):
    from forcepho_b200.patches.device_store import REGION_DTYPE
    from forcepho_b200.region import REGION_CIRCLE
    recs = np.zeros(len(idx), dtype=REGION_DTYPE)
    recs["kind"] = REGION_CIRCLE
    for r in recs:
        r["p"][:3] = (*rng.uniform(0.2 * nside, 0.8 * nside, 2), rng.choice(radii) ** 2)
    return recs


@pytest.mark.parametrize("s,nside", [(8, 512), (4, 256), (6, 300), (3, 192), (16, 512)])
@pytest.mark.parametrize("n", [1, 3, 70])
def test_gather_equals_numpy(s, nside, n):
    st, exps, rng = store(s, nside, min(n, 4), seed=s + n)
    idx = rng.integers(0, len(exps), n).astype(np.int32)
    recs = circles(idx, nside, [0.0, 0.3, 2.5 * s, 9.0 * s, 40.0 * s], rng)
    for bg, max_snr in ((None, 0.0), (rng.normal(0, 0.01, n).astype(np.float32), 100.0)):
        pix, start, cnt = st.gather(idx, recs, background=bg, max_snr=max_snr)
        want, n_want = pack_numpy(exps, idx, recs, s, bg, max_snr)
        np.testing.assert_array_equal(cnt, n_want)
        np.testing.assert_array_equal(start, np.concatenate([[0], np.cumsum(n_want)[:-1]]))
        for a, b in zip(pix, want):
            np.testing.assert_array_equal(a.cpu().numpy(), b)
        again, _, _ = st.gather(idx, recs, background=bg, max_snr=max_snr,
                                npix=int(n_want.sum()))
        for a, b in zip(again, want):
            np.testing.assert_array_equal(a.cpu().numpy(), b)
    st.free()


def test_gather_halves():
    """A ticket is good once, and not after another count."""
    import torch
    from forcepho_b200 import _lib
    st, exps, rng = store(8, 256, 2)
    idx = np.array([0, 1], dtype=np.int32)
    recs = circles(idx, 256, [30.0], rng)
    npix, ticket = ctypes.c_int64(), ctypes.c_uint64()

    def begin():
        _lib.call("fpho_store_gather_begin", st.handle, 2, idx.ctypes.data, recs.ctypes.data,
                  ctypes.byref(npix), ctypes.byref(ticket), None)

    begin()
    bufs = [torch.zeros(npix.value, device="cuda") for _ in range(4)]
    start, n = np.zeros(2, np.int32), np.zeros(2, np.int32)

    def end():
        _lib.call("fpho_store_gather_end", st.handle, ticket, 2, None, 0.0,
                  *[b.data_ptr() for b in bufs], npix.value, start.ctypes.data, n.ctypes.data, None)

    end()
    want, n_want = pack_numpy(exps, idx, recs, 8, None, 0.0)
    np.testing.assert_array_equal(n, n_want)
    for a, b in zip(bufs, want):
        np.testing.assert_array_equal(a.cpu().numpy(), b)
    for between in (lambda: None, lambda: (begin(), st.count(idx, recs))):
        between()
        with pytest.raises(_lib.FphoError) as exc:
            end()
        assert exc.value.code == _lib.FPHO_ERR_STATE
    st.free()


@pytest.mark.parametrize("n_exp", [0, 1, 3])
def test_gather_halves_of_different_lengths_are_refused(n_exp):
    import torch
    from forcepho_b200 import _lib
    st, _, rng = store(8, 256, 4)
    idx = np.arange(4, dtype=np.int32)
    st.count(idx, circles(idx, 256, [30.0], rng))      # four exposures' totals are about
    npix, ticket = ctypes.c_int64(), ctypes.c_uint64()
    recs = circles(idx[:2], 256, [30.0], rng)
    _lib.call("fpho_store_gather_begin", st.handle, 2, idx.ctypes.data, recs.ctypes.data,
              ctypes.byref(npix), ctypes.byref(ticket), None)
    bufs = [torch.zeros(npix.value, device="cuda") for _ in range(4)]
    start, n = np.zeros(4, np.int32), np.zeros(4, np.int32)
    with pytest.raises(_lib.FphoError, match="exposures were counted"):
        _lib.call("fpho_store_gather_end", st.handle, ticket, n_exp, None, 0.0,
                  *[b.data_ptr() for b in bufs], npix.value, start.ctypes.data, n.ctypes.data,
                  None)
    st.free()
