"""The many-row projection's input conversion where its threads' rounds end: one chunk a thread and several, rows that are re-read
(longer than the threads keep), the splits' sums, padding rows. Every converted half against numpy."""
import ctypes

import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,norm,splits", [(1, 256, True, 0), (17, 1024, False, 0), (33, 6144, True, 3), (20, 6400, False, 9), (128, 5120, True, 7),
                                                (16, 17408, False, 0), (19, 18432, True, 1), (3, 33024, True, 2), (130, 512, True, 0)])
def test_converted_rows(rows, k, norm, splits):
    from splash_b200 import lib
    lib.init(0)
    l = lib.ops()
    P, U = ctypes.c_void_p, ctypes.c_uint32
    l.sb_linear_wide_prepare_sum.argtypes = [P, P, U, U, P, U, P, U, U, U, P, P, U]
    rng = np.random.default_rng(rows * 31 + k)
    x = ol.f2bf((rng.standard_normal((rows, k)) * np.exp2(rng.integers(-20, 20, (rows, 1)))).astype(np.float32))
    w = rng.uniform(0.5, 1.5, k).astype(np.float32)
    xd, wd = lib.DeviceBuffer.from_numpy(x), lib.DeviceBuffer.from_numpy(w)
    out = lib.DeviceBuffer(int(l.sb_linear_wide_prepared_bytes(rows, k)))
    if splits:
        part = (rng.standard_normal((splits, rows, k)) * np.abs(ol.bf2f(x)).max(axis=1)[None, :, None]).astype(np.float32)
        pd, sd = lib.DeviceBuffer.from_numpy(part), lib.DeviceBuffer(rows * k * 2 + 256)
        lib.check(l.sb_linear_wide_prepare_sum(None, pd.ptr, splits, k, xd.ptr, k, sd.ptr, k, rows, k, wd.ptr if norm else None, out.ptr, 0))
        total = part[0].copy()
        for s in range(1, splits):
            total += part[s]                       # in split order, fp32
        x = ol.f2bf(total + ol.bf2f(x))
        assert np.array_equal(sd.to_numpy(np.uint16, (rows, k)), x)
    else:
        lib.check(l.sb_linear_wide_prepare(None, xd.ptr, rows, k, k, wd.ptr if norm else None, out.ptr, 0))
    lib.stream_sync()
    v = ol.bf2f(x).astype(np.float64)
    if norm:
        v = v / np.sqrt((v * v).mean(axis=1, keepdims=True) + 1e-6) * w
    passes, per_pass = (rows + 127) // 128, int(l.sb_linear_wide_prepared_bytes(128, k))
    order = np.array([0, 2, 1, 3, 4, 6, 5, 7])
    for ps in range(passes):
        n = min(128, rows - 128 * ps)
        padded = (n + 15) // 16 * 16
        raw = out.to_numpy(np.uint8, (1024 + padded * k * 2,), offset=ps * per_pass)
        scale = raw[:4 * padded].view(np.float32)
        halves = raw[1024:].view(np.float16).reshape(k // 64, 4, padded // 8, 2, 8, 8)  # [64 inputs][16 inputs][8 rows][8 inputs][row][input]
        got = halves.transpose(2, 4, 0, 1, 3, 5).reshape(padded, k // 8, 8)
        got = got[:, :, np.argsort(order)].reshape(padded, k).astype(np.float64) * scale[:, None]
        want = v[128 * ps:128 * ps + n]
        # without a norm the halves are the bf16 values themselves (exact down to 2^-24 of the row's largest); with it one rounding to
        # bf16 of a product whose statistics carry fp32 sums
        tol = np.abs(want) * (2.0 ** -7 if norm else 0.0) + np.abs(want).max(axis=1, keepdims=True) * 2.0 ** -24
        assert (np.abs(got[:n] - want) <= tol).all()
        assert not got[n:].any() and np.array_equal(np.log2(scale[:n]), np.round(np.log2(scale[:n])))
