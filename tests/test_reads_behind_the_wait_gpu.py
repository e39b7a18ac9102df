"""Launches that follow one another without a synchronisation, each allowed to start while the one ahead drains: what the kernel ahead
writes is what the next one reads, weights included (only a cell that the caller vouches for may be read early)."""
import ctypes

import numpy as np
import pytest

import oracle_lib as ol
import quant_fixtures as qf
from test_ops_gpu import _gdn_inputs, _setup

pytestmark = pytest.mark.gpu


def _project(lib, w, x, out, n, k, f32):
    lib.linear(w.ptr, x.ptr, out.ptr, lib.FMT_Q4K, n, k, 16, out_f32=f32, flags=lib.LINEAR_PDL)


def test_norm_weights_written_by_the_launch_ahead():
    lib, l, _ = _setup()
    n, k, rows = 5120, 17408, 48
    w, x = (lib.DeviceBuffer.from_numpy(a) for a in (qf.realistic(0, n, k, seed=1), qf.activations(16, k, seed=2)))
    rowsd = lib.DeviceBuffer.from_numpy(qf.activations(rows, n, seed=3))
    norm, stale = lib.DeviceBuffer(16 * n * 4), np.full(16 * n, 7.0, np.float32)
    size = int(l.sb_linear_wide_prepared_bytes(rows, n))
    behind, after = lib.DeviceBuffer(size), lib.DeviceBuffer(size)
    for b in (behind, after):
        b.fill(0)
    for _ in range(10):
        norm.upload(stale)
        lib.stream_sync()
        _project(lib, w, x, norm, n, k, True)
        lib.check(l.sb_linear_wide_prepare(None, rowsd.ptr, rows, n, n, norm.ptr, behind.ptr, lib.LINEAR_PDL))
        lib.stream_sync()
        lib.check(l.sb_linear_wide_prepare(None, rowsd.ptr, rows, n, n, norm.ptr, after.ptr, 0))
        lib.stream_sync()
        assert np.array_equal(behind.to_numpy(np.uint8, (size,)), after.to_numpy(np.uint8, (size,)))


def test_gate_weights_written_by_the_launch_ahead():
    lib, l, _ = _setup()
    rng = np.random.default_rng(5)
    KH, VH, n, k = 4, 48, 64, 17408
    x = _gdn_inputs(rng, KH, VH)
    VW, C, KW = x["VW"], x["C"], x["KW"]
    d = {name: lib.DeviceBuffer.from_numpy(x[name]) for name in ("qkvz", "b", "a", "conv_w", "norm_w", "cs", "state")}
    w = lib.DeviceBuffer.from_numpy(qf.realistic(0, n, k, seed=1))
    small = lib.DeviceBuffer.from_numpy(ol.f2bf(ol.bf2f(qf.activations(16, k, seed=2)) * np.float32(0.01)))
    scale, bias = lib.DeviceBuffer(16 * n * 4), lib.DeviceBuffer(16 * n * 2)
    step = {name: lib.DeviceBuffer(size) for name, size in dict(inputs=16 * C * 2, k=16 * KW * 2, v=16 * VW * 2, beta=16 * VH * 2, decay=16 * VH * 4).items()}
    cs, state, hidden = lib.DeviceBuffer(x["cs"].nbytes), lib.DeviceBuffer(x["state"].nbytes), lib.DeviceBuffer(16 * VW * 2)
    args = lib.SbGdnArgs(d["qkvz"].ptr, d["b"].ptr, d["a"].ptr, d["conv_w"].ptr, scale.ptr, bias.ptr, d["norm_w"].ptr, d["cs"].ptr, cs.ptr, d["state"].ptr,
                         state.ptr, lib.SbGdnTape(), lib.SbGdnTape(*(step[name].ptr for name in ("inputs", "k", "v", "beta", "decay"))), hidden.ptr, None,
                         16, 0, KH, VH, x["stride"], VH, VW, 0)
    read = lambda: (step["decay"].to_numpy(np.uint32, (16, VH)), hidden.to_numpy(np.uint16, (16, VW)))
    for ahead in ("scale", "bias"):
        for _ in range(10):
            scale.upload(np.full(16 * n, -3.0, np.float32))
            bias.upload(ol.f2bf(np.full(16 * n, 2.0, np.float32)))
            lib.stream_sync()
            _project(lib, w, small, scale if ahead == "scale" else bias, n, k, ahead == "scale")
            lib.check(l.sb_gdn_verify(None, ctypes.byref(args)))
            lib.stream_sync()
            behind = read()
            lib.check(l.sb_gdn_verify(None, ctypes.byref(args)))
            lib.stream_sync()
            for a, b in zip(behind, read()):
                assert np.array_equal(a, b)
