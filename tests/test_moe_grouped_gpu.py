"""MoE blocks of many rows where the grouping and the combine end: the most routes a launch takes, one more, rows that lie on four
bytes only (on eight where the sums stay fp32)."""
import ctypes

import numpy as np
import pytest

import oracle_lib as ol
import quant_fixtures as qf
from test_ops_gpu import P, _setup, ulp_bf16

pytestmark = pytest.mark.gpu


def _block(lib, l, rows, routes, experts, H, I, seed):
    rng = np.random.default_rng(seed)
    x, res = (ol.f2bf(rng.standard_normal((rows, H)).astype(np.float32)) for _ in range(2))
    h = dict(x=x, res=res, selected=rng.integers(0, experts, (rows, routes)).astype(np.uint32), weights=rng.uniform(0.02, 0.1, (rows, routes)).astype(np.float32),
             gate=qf.realistic(0, experts * I, H, seed=1), up=qf.realistic(0, experts * I, H, seed=2), down=qf.realistic(0, experts * H, I, seed=3))
    d = {k: lib.DeviceBuffer.from_numpy(v) for k, v in h.items()}
    scratch = lib.DeviceBuffer(int(l.sb_moe_scratch_bytes(rows, routes, H, I)))
    args = lambda out, res_ptr=None: lib.SbMoeExpertArgs(d["x"].ptr, res_ptr or d["res"].ptr, d["selected"].ptr, d["weights"].ptr, d["gate"].ptr, d["up"].ptr, d["down"].ptr,
                                                         scratch.ptr, out, rows, routes, H, I, lib.FMT_Q4K, experts)
    return h, d, scratch, args


def test_the_most_routes():
    lib, l, o = _setup()
    rows, routes, experts, H, I = 512, 32, 7, 256, 256
    h, d, scratch, args = _block(lib, l, rows, routes, experts, H, I, 5)
    out = lib.DeviceBuffer(rows * H * 2)
    lib.check(l.sb_moe_experts(None, ctypes.byref(args(out.ptr))))
    lib.stream_sync()
    assert lib.device_status() == 0
    want, y64 = np.zeros((rows, H), np.uint16), np.zeros((rows * routes, H), np.float64)
    assert o.so_moe_experts(*(P(h[k]) for k in ("x", "res", "selected", "weights", "gate", "up", "down")), rows, routes, H, I, experts, P(want), P(y64)) == 0
    y = np.abs(y64.reshape(rows, routes, H))
    # (weights rounded to half, the intermediate rows and the routes' results to bf16)
    slack = (h["weights"][:, :, None] * (ulp_bf16(y) + 2.0 ** -6 * y.mean(axis=2, keepdims=True))).sum(axis=1)
    g, w = (ol.bf2f(a).astype(np.float64) for a in (out.to_numpy(np.uint16, (rows, H)), want))
    assert (np.abs(g - w) <= 2 * ulp_bf16(w) + slack).all()
    too_many = args(out.ptr)
    too_many.rows = 513
    assert l.sb_moe_experts(None, ctypes.byref(too_many)) == -1


def test_rows_on_four_bytes_give_the_same_bits():
    lib, l, _ = _setup()
    rows, routes, experts, H, I = 21, 5, 9, 512, 256
    h, d, scratch, args = _block(lib, l, rows, routes, experts, H, I, 6)
    res = lib.DeviceBuffer(rows * H * 2 + 16)
    res.upload(h["res"], offset=4)
    got = []
    for off, res_ptr in ((0, None), (4, None), (0, res.ptr + 4), (12, res.ptr + 4)):
        out = lib.DeviceBuffer(rows * H * 2 + 16)
        lib.check(l.sb_moe_experts(None, ctypes.byref(args(out.ptr + off, res_ptr))))
        lib.stream_sync()
        got.append(out.to_numpy(np.uint16, (rows, H), offset=off))
    for g in got[1:]:
        assert np.array_equal(g, got[0])
    u = ctypes.c_uint32
    l.sb_moe_experts_partial.argtypes = [ctypes.c_void_p, ctypes.c_void_p, u, u, u, u, u]
    sums = []
    for off in (0, 8):
        out = lib.DeviceBuffer(rows * H * 4 + 16)
        a = args(out.ptr + off)
        lib.check(l.sb_moe_experts_partial(None, ctypes.byref(a), 0, experts, 0xFFFFFFFF, 0, rows))
        lib.stream_sync()
        sums.append(out.to_numpy(np.float32, (rows, H), offset=off))
    assert lib.device_status() == 0
    assert np.array_equal(*sums)
    assert np.array_equal(ol.f2bf(ol.bf2f(h["res"]) + sums[0]), got[0])
