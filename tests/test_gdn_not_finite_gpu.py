"""An infinity or NaN in one row of a Gated-DeltaNet step stays with the rows whose path it lies on: the rows before it in a chain,
the other branches of a tree and the other lanes keep every bit."""
import ctypes

import numpy as np
import pytest

from test_ops_gpu import _gdn_inputs, _setup, _tree_rows

pytestmark = pytest.mark.gpu

KH, VH, D = 2, 6, 128
BRANCHES = [0, 0, 1, 2, 0, 4, 5, 4, 2, 8, 9, 10, 0, 12, 13, 14]


def _step(lib, l, x, lanes, tree, rows):
    """One step of `lanes` lanes, each holding the rows of x (lane 0 those of x['qkvz'], the others of x['clean'])."""
    up = lib.DeviceBuffer.from_numpy
    C, KW, VW = x["C"], x["KW"], x["VW"]
    rep = lambda a: np.concatenate([a] * lanes)
    d = {n: up(rep(x[n]) if n in ("cs", "state") else x[n]) for n in ("conv_w", "a_scale", "dt_bias", "norm_w", "cs", "state")}
    for n in ("qkvz", "b", "a"):
        d[n] = up(np.concatenate([x[n]] + [x["clean"][n]] * (lanes - 1)))
    p = {n: up(rep(v)) for n, v in x["pend"].items()}
    s = {n: lib.DeviceBuffer(lanes * size) for n, size in dict(inputs=16 * C * 2, k=16 * KW * 2, v=16 * VW * 2, beta=16 * VH * 2, decay=16 * VH * 4).items()}
    cs, st, hid = lib.DeviceBuffer(lanes * x["cs"].nbytes), lib.DeviceBuffer(lanes * x["state"].nbytes), lib.DeviceBuffer(lanes * 16 * VW * 2)
    hid.fill(0)
    tape = lambda t: lib.SbGdnTape(*(t[n].ptr for n in ("inputs", "k", "v", "beta", "decay")))
    a = lib.SbGdnArgs(d["qkvz"].ptr, d["b"].ptr, d["a"].ptr, d["conv_w"].ptr, d["a_scale"].ptr, d["dt_bias"].ptr, d["norm_w"].ptr, d["cs"].ptr, cs.ptr,
                      d["state"].ptr, st.ptr, tape(p), tape(s), hid.ptr, None, rows, 3, KH, VH, x["stride"], VH, VW, 0)
    a.lanes = lanes if lanes > 1 else 0
    if tree is not None:
        t = up(np.concatenate([np.pad(tree, ((0, 16 - rows), (0, 0)))] * lanes))
        a.tree = t.ptr
    lib.check(l.sb_gdn_verify(None, ctypes.byref(a)))
    lib.stream_sync()
    assert lib.device_status() == 0
    return hid.to_numpy(np.uint16, (lanes, 16, VW)), st.to_numpy(np.uint32, (lanes,) + x["state"].shape)


@pytest.mark.parametrize("what,value", [("value", 0x7F80), ("value", 0x7FC0), ("key", 0x7FC0), ("query", 0x7FC0), ("beta", 0x7FC0), ("decay", 0x7FC0)])
@pytest.mark.parametrize("shape,at,rows", [("chain", 3, 16), ("chain", 14, 15), ("chain", 1, 2), ("tree", 1, 16), ("tree", 8, 16), ("tree", 4, 13)])
@pytest.mark.parametrize("lanes", [1, 2])
def test_a_row_that_is_not_finite_stays_on_its_path(what, value, shape, at, rows, lanes):
    lib, l, _ = _setup()
    x = _gdn_inputs(np.random.default_rng(at * 16 + rows), KH, VH)
    tree = _tree_rows(BRANCHES[:rows]) if shape == "tree" else None
    x["clean"] = {n: x[n] for n in ("qkvz", "b", "a")}
    want, want_state = _step(lib, l, x, lanes, tree, rows)
    for n in ("qkvz", "b", "a"):
        x[n] = x[n].copy()
    KW = x["KW"]
    if what in ("beta", "decay"):
        x["b" if what == "beta" else "a"][at] = value
    else:
        c0 = {"query": 0, "key": KW, "value": 2 * KW}[what]
        x["qkvz"][at, c0 + 5::D][:] = value
    got, got_state = _step(lib, l, x, lanes, tree, rows)
    clear = np.ones((lanes, 16), bool)
    for r in range(rows):
        clear[0, r] = not (int(tree[r, 0]) >> at & 1 if shape == "tree" else r >= at)
    assert 0 < clear[0, :rows].sum() < rows
    assert np.array_equal(got[clear], want[clear])
    assert np.array_equal(got_state, want_state)  # (the block's own rows are never folded here)
