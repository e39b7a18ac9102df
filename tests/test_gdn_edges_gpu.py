"""The Gated-DeltaNet kernel where its eights, sixteens and quarters end: every kind of row and pending count, chains and trees,
tapes and cells that lie on their element's two bytes only. Against the CPU oracle, which advances the state row by row."""
import ctypes

import numpy as np
import pytest

import oracle_lib as ol
from test_ops_gpu import _setup, _tree_rows, check_gdn_hidden, gdn_case, ulp_bf16

pytestmark = pytest.mark.gpu


def _check(got, want, rows):
    assert np.array_equal(got["cs"], want["cs"])
    assert np.array_equal(got["inputs"][:rows], want["inputs"][:rows])
    for n in ("k", "v", "beta"):
        g, w = ol.bf2f(got[n][:rows]).astype(np.float64), ol.bf2f(want[n][:rows]).astype(np.float64)
        assert (np.abs(g - w) <= 3 * ulp_bf16(w)).all(), n
    # fp32 sums of up to 16 rank-1 updates over 128 columns: 2^-23 times a few dozen operations on values of the state's size
    assert np.abs(got["state"] - want["state"]).max() <= 1e-5 * np.abs(want["state"]).max()
    if rows:
        check_gdn_hidden(got["hidden"][:rows], want["hidden"][:rows])


@pytest.mark.parametrize("rows,pending", [(0, 16), (1, 0), (1, 16), (7, 1), (8, 8), (9, 9), (15, 15), (16, 0), (16, 1)])
def test_rows_and_pending_rows(rows, pending):
    lib, l, o = _setup()
    got, want, _ = gdn_case(lib, l, o, key_heads=2, value_heads=6, rows=rows, pending_rows=pending, tiled=True, seed=100 + 17 * rows + pending)
    _check(got, want, rows)


@pytest.mark.parametrize("shape", ["star", "pairs", "late"])
def test_trees_over_sparse_pending_paths(shape):
    lib, l, o = _setup()
    parent = {"star": [0] * 16, "pairs": [0] + [max(0, (r - 1) // 2) for r in range(1, 16)], "late": [0, 0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 0, 14]}[shape]
    got, want, rows = gdn_case(lib, l, o, key_heads=4, value_heads=4, rows=16, pending_rows=0, tiled=False, seed=len(shape), tree=_tree_rows(parent),
                               pending_path=0b1000000010000001)
    _check(got, want, rows)


def test_tape_on_two_byte_boundaries_gives_the_same_bits():
    """The step's tape and the carried convolution rows are written eight channels at a time where they may be; a tape two bytes
    off gets the same values."""
    lib, l, _ = _setup()
    rng = np.random.default_rng(7)
    KH, VH, D, rows = 2, 4, 128, 11
    KW, VW = KH * D, VH * D
    C = 2 * KW + VW
    bf = lambda shape, s: ol.f2bf((rng.standard_normal(shape) * s).astype(np.float32))
    up = lib.DeviceBuffer.from_numpy
    d = dict(qkvz=up(bf((16, C + VW), 1.0)), b=up(bf((16, VH), 1.0)), a=up(bf((16, VH), 1.0)), conv_w=up(bf((C, 4), 0.4)),
             a_scale=up((-np.exp(rng.uniform(-3, 0.5, VH))).astype(np.float32)), dt=up(bf((VH,), 0.5)), norm=up(np.ones(D, np.float32)),
             cs=up(bf((3, C), 1.0)), state=up((rng.standard_normal((VH, D, D)) * 0.05).astype(np.float32)))
    results = []
    for off in (0, 2):
        t = {n: lib.DeviceBuffer(16 * w * 2 + 256) for n, w in (("inputs", C), ("k", KW), ("v", VW), ("beta", VH))}
        decay, cs, st, hid = lib.DeviceBuffer(16 * VH * 4), lib.DeviceBuffer(3 * C * 2 + 256), lib.DeviceBuffer(VH * D * D * 4), lib.DeviceBuffer(16 * VW * 2)
        args = lib.SbGdnArgs(d["qkvz"].ptr, d["b"].ptr, d["a"].ptr, d["conv_w"].ptr, d["a_scale"].ptr, d["dt"].ptr, d["norm"].ptr, d["cs"].ptr, cs.ptr + off,
                             d["state"].ptr, st.ptr, lib.SbGdnTape(), lib.SbGdnTape(t["inputs"].ptr + off, t["k"].ptr + off, t["v"].ptr + off, t["beta"].ptr + off, decay.ptr),
                             hid.ptr, None, rows, 0, KH, VH, C + VW, VH, VW, 0)
        lib.check(l.sb_gdn_verify(None, ctypes.byref(args)))
        lib.stream_sync()
        assert lib.device_status() == 0
        out = [t[n].to_numpy(np.uint16, (rows, w), offset=off) for n, w in (("inputs", C), ("k", KW), ("v", VW), ("beta", VH))]
        results.append(out + [cs.to_numpy(np.uint16, (3, C), offset=off), hid.to_numpy(np.uint16, (rows, VW)), st.to_numpy(np.float32, (VH, D, D))])
    for x, y in zip(*results):
        assert np.array_equal(x, y)
