"""The experts' kernels of one lane's block where their groups of eight and their tiles end: one route in all, every route to one
expert, as many routes as a block may have, the narrowest widths, rows that start on two bytes only, ids past the experts.
Against the oracle's fp64 statement."""
import ctypes

import numpy as np
import pytest

import oracle_lib as ol
import quant_fixtures as qf
from test_ops_gpu import P, _setup, ulp_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,routes,experts,H,I,choice,offset", [
    (1, 1, 1, 256, 256, "one", 0),          # (experts of up to 1024 x 512 and few routes: a matrix-vector product a route)
    (16, 1, 3, 512, 256, "one", 0),
    (9, 2, 4, 1024, 256, "spread", 2),      # the most weights of such a block
    (1, 1, 1, 1280, 256, "one", 0),
    (16, 1, 3, 1280, 256, "one", 0),        # sixteen routes of one expert: two full groups
    (10, 2, 4, 1024, 256, "spread", 2),     # one route too many for it
    (9, 2, 4, 256, 768, "one", 2),          # nine and nine: a group of eight and one of one
    (16, 32, 40, 512, 512, "spread", 0),    # the most routes
    (5, 7, 300, 768, 256, "spread", 6),
    (3, 4, 6, 512, 256, "past", 0),         # an id past the experts reads the last one, as ever
    (3, 4, 6, 1280, 256, "past", 0),
    (2, 3, 5, 256, 2304, "spread", 0),      # an intermediate row of more than one round of its conversion
])
def test_few_rows_experts(rows, routes, experts, H, I, choice, offset):
    lib, l, o = _setup()
    rng = np.random.default_rng(rows * 100 + routes)
    kinds = min(experts, 6)  # (experts share a few tensors; the ids still differ)
    pool = lambda n, k, seed: [qf.realistic(0, n, k, seed=seed + e) for e in range(kinds)]
    gate, up, down = ([t[e % kinds] for e in range(experts)] for t in (pool(I, H, 1), pool(I, H, 50), pool(H, I, 90)))
    gate, up, down = (np.concatenate(t) for t in (gate, up, down))
    x, res = (ol.f2bf(rng.standard_normal((rows, H)).astype(np.float32)) for _ in range(2))
    selected = np.zeros((rows, routes), np.uint32)
    if choice == "one":
        selected[:] = experts - 1
    else:
        selected[:] = rng.integers(0, experts, (rows, routes))
    if choice == "past":
        selected[1, 2] = experts + 5
    weights = rng.uniform(0.05, 0.6, (rows, routes)).astype(np.float32)
    xd = lib.DeviceBuffer(x.nbytes + 256)
    xd.upload(x, offset=offset)
    sd, wd, rd = (lib.DeviceBuffer.from_numpy(a) for a in (selected, weights, res))
    gd, ud, dd = (lib.DeviceBuffer.from_numpy(a) for a in (gate, up, down))
    scratch, out = lib.DeviceBuffer(int(l.sb_moe_scratch_bytes(rows, routes, H, I))), lib.DeviceBuffer(rows * H * 2 + 256)
    ea = lib.SbMoeExpertArgs(xd.ptr + offset, rd.ptr, sd.ptr, wd.ptr, gd.ptr, ud.ptr, dd.ptr, scratch.ptr, out.ptr, rows, routes, H, I, lib.FMT_Q4K, experts)
    for _ in range(2):  # the second call finds the first one's groups in the scratch
        lib.check(l.sb_moe_experts(None, ctypes.byref(ea)))
    lib.stream_sync()
    assert lib.device_status() == 0
    want, y64 = np.zeros((rows, H), np.uint16), np.zeros((rows * routes, H), np.float64)
    assert o.so_moe_experts(P(x), P(res), P(np.minimum(selected, experts - 1)), P(weights), P(gate), P(up), P(down), rows, routes, H, I, experts, P(want), P(y64)) == 0
    # A route's result is rounded to bf16 before its weight, so is the intermediate row: half an ulp of each route's value, times its
    # weight, may move either way, beside the result's own rounding.
    y = y64.reshape(rows, routes, H)
    slack = (np.abs(weights)[:, :, None] * (ulp_bf16(y) + 2e-3 * np.abs(y).mean(axis=2, keepdims=True))).sum(axis=1)
    g, w = (ol.bf2f(a).astype(np.float64) for a in (out.to_numpy(np.uint16, (rows, H)), want))
    assert (np.abs(g - w) <= 2 * ulp_bf16(w) + slack).all()
