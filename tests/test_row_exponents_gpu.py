"""Rows at both ends of bf16's range through every conversion that takes a power of two out of a row: the 16-row and the many-row
projection, the MoE block of a few rows and of many. A row of the smallest magnitudes beside zeros is not NaN, a finite row of
the largest is not infinite."""
import ctypes

import numpy as np
import pytest

import oracle_lib as ol
import quant_fixtures as qf
from test_linear_gpu import run_linear
from test_ops_gpu import P, _setup, ulp_bf16

pytestmark = pytest.mark.gpu

POWERS = (-133, -126, -119, -118, -117, -116, 100, 126, 127)


def _weights(n, k, seed):
    """Q4_K rows of values below 0.06, so that a product with a row of the largest magnitudes stays finite."""
    rng = np.random.default_rng(seed)
    return qf.q4k_blocks(rng, n, k, rng.uniform(2e-5, 6e-5, (n, k // 256)), rng.uniform(2e-5, 6e-5, (n, k // 256)))


def _rows(rng, rows, k, exponent):
    """bf16 rows that are zero but for forty values of up to 2^exponent times 1.99."""
    x = np.zeros((rows, k), np.float64)
    for r in range(rows):
        at = rng.permutation(k)[:40]
        x[r, at] = np.ldexp(rng.uniform(0.5, 1.99, 40) * rng.choice([-1, 1], 40), exponent)
        x[r, at[0]] = np.ldexp(1.0, exponent)
    return ol.f2bf(x.astype(np.float32))


@pytest.mark.parametrize("rows", [16, 40])
@pytest.mark.parametrize("exponent", POWERS)
def test_projection(rows, exponent):
    lib, l, o = _setup()
    n, k = 256, 1024
    X, W = _rows(np.random.default_rng(rows), rows, k, exponent), _weights(n, k, 3)
    got = run_linear(lib, 0, W, n, k, X, rows, out_f32=True).astype(np.float64)
    w, x = ol.dequant(o, 0, W, n, k).astype(np.float64), ol.bf2f(X).astype(np.float64)
    want = x @ w.T
    # weights may be rounded to half (three roundings of 2^-11), a result below fp32's normal range to 2^-149
    bound = 2.0 ** -9 * (np.abs(x) @ np.abs(w).T) + 2.0 ** -14 * np.abs(x).sum(axis=1, keepdims=True) * np.abs(w).max() + 2.0 ** -148
    assert np.isfinite(got).all() and (np.abs(got - want) <= bound).all()


@pytest.mark.parametrize("rows,H", [(3, 512), (3, 1280), (24, 512)])
@pytest.mark.parametrize("exponent", POWERS + (-57, -54))
def test_moe_block(rows, H, exponent):
    """2^-57 and 2^-54: rows whose SwiGLU products, not they themselves, lie where a row's power of two ends."""
    lib, l, o = _setup()
    rng = np.random.default_rng(rows)
    routes, experts, I = 2, 3, 256
    gate, down = _weights(experts * I, H, 1), _weights(experts * H, I, 2)
    up = _weights(experts * I, H, 4)
    if exponent > 0:
        up[:] = 0  # (the product of two rows of 2^100 would be infinite; the down projection then reads zeros)
    x = _rows(rng, rows, H, exponent)
    res = ol.f2bf(np.zeros((rows, H), np.float32) if exponent < 0 else rng.standard_normal((rows, H)).astype(np.float32))
    selected = rng.integers(0, experts, (rows, routes)).astype(np.uint32)
    weights = rng.uniform(0.2, 0.6, (rows, routes)).astype(np.float32)
    xd, sd, wd, rd, gd, ud, dd = (lib.DeviceBuffer.from_numpy(a) for a in (x, selected, weights, res, gate, up, down))
    scratch, out = lib.DeviceBuffer(int(l.sb_moe_scratch_bytes(rows, routes, H, I))), lib.DeviceBuffer(rows * H * 2)
    a = lib.SbMoeExpertArgs(xd.ptr, rd.ptr, sd.ptr, wd.ptr, gd.ptr, ud.ptr, dd.ptr, scratch.ptr, out.ptr, rows, routes, H, I, lib.FMT_Q4K, experts)
    lib.check(l.sb_moe_experts(None, ctypes.byref(a)))
    lib.stream_sync()
    assert lib.device_status() == 0
    want, y64 = np.zeros((rows, H), np.uint16), np.zeros((rows * routes, H), np.float64)
    assert o.so_moe_experts(P(x), P(res), P(selected), P(weights), P(gate), P(up), P(down), rows, routes, H, I, experts, P(want), P(y64)) == 0
    g, w = (ol.bf2f(b).astype(np.float64) for b in (out.to_numpy(np.uint16, (rows, H)), want))
    # a route's result and its intermediate row are rounded to bf16, many rows' weights to half; below the normal range of bf16
    # by half of its smallest step, a route's each
    y = np.abs(y64.reshape(rows, routes, H))
    slack = (np.abs(weights)[:, :, None] * (2.0 ** -6 * y + 2.0 ** -6 * y.mean(axis=2, keepdims=True))).sum(axis=1) + 2.0 ** -133 * (1 + routes)
    assert np.isfinite(g).all() and (np.abs(g - w) <= 2 * ulp_bf16(w) + slack).all()
