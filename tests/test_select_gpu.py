"""The cluster selection kernel (sb_select.cuh) at the sizes where it can go wrong: vocabularies around its shards of 256 ids, its
eight slices, its limit and the one-block kernel above it; logits with ties, holes and a flat row; every end of the
distribution. Against the CPU oracle, which walks the distribution by its definition."""
import ctypes

import numpy as np
import pytest

import oracle_lib as ol
from oracle_lib import ptr as P

pytestmark = pytest.mark.gpu

POLICIES = [(0.0, 0, 1.0), (0.05, 0, 1.0), (0.0, 40, 1.0), (0.0, 0, 0.6), (0.01, 300, 0.9), (0.0, 5000, 0.999)]


def _logits(rng, rows, vocab):
    x = (rng.standard_normal((rows, vocab)) * 3).astype(np.float32)
    if rows > 1:
        x[1] = np.round(x[1] * 2) / 2                    # many ties
    if rows > 2:
        x[2, ::3] = -np.inf                              # holes
        x[2, 1::7] = np.nan
        x[2, vocab // 2] = 4.0
    if rows > 3:
        x[3] = 1.5                                       # flat
    if rows > 4:
        x[4] = np.nan                                    # nothing selectable
    return x


@pytest.mark.parametrize("vocab", [1, 255, 257, 2048, 2049, 50257, 262144, 262145])
def test_selection_at_the_cluster_kernels_edges(vocab):
    from splash_b200 import lib
    lib.init(0)
    l, o = lib.ops(), ol.bind_ops(ol.load())
    rows, T = 6, 0.8
    rng = np.random.default_rng(vocab)
    logits = _logits(rng, rows, vocab)
    inputs = np.concatenate([[0], np.nan_to_num(logits, nan=-1e30).argmax(axis=1)[:-1]]).astype(np.uint32)
    uniforms = rng.random(80).astype(np.float32)
    ld, idd, ud = (lib.DeviceBuffer.from_numpy(x) for x in (logits, inputs, uniforms))
    sd, cd = lib.DeviceBuffer(rows * 4), lib.DeviceBuffer(rows * 8)
    wd = lib.DeviceBuffer(int(l.sb_sample_workspace_bytes(rows, vocab)))
    for temperature, (min_p, top_k, top_p) in [(0.0, POLICIES[0])] + [(T, p) for p in POLICIES]:
        a = lib.SbSampleArgs(ld.ptr, idd.ptr, ud.ptr, sd.ptr, wd.ptr, rows, vocab, vocab, temperature, min_p, top_k, top_p, cd.ptr)
        filtered = min_p > 0 or 0 < top_k < vocab or top_p < 1
        if vocab > 262144 and filtered:
            assert l.sb_sample_verify(None, ctypes.byref(a)) == -1   # the ends' limit, as ever
            continue
        lib.check(l.sb_sample_verify(None, ctypes.byref(a)))
        got, gcut = sd.to_numpy(np.uint32, (rows,)), cd.to_numpy(np.uint32, (rows, 2))
        assert lib.device_status() == 0
        want, margin, wcut = np.zeros(rows, np.uint32), np.zeros(rows, np.float64), np.zeros((rows, 2), np.uint32)
        if temperature == 0.0:
            o.so_sample_verify(P(logits), vocab, vocab, rows, P(inputs), 0.0, None, P(want), None)
            assert np.array_equal(got, want)
            continue
        o.so_sample_verify_filtered(P(logits), vocab, vocab, rows, P(inputs), T, min_p, top_k, top_p, P(uniforms), P(want), P(margin), P(wcut))
        assert got[4] == want[4] == 0xFFFFFFFF
        live = np.arange(rows) != 4
        # Weights come from two expf's (2 ulp apart), masses from sums of up to 2^18 of them in one order: an end moves only where a
        # mass lies within 2^-19 of the nucleus, a selection only where its test does (margin, relative).
        same = (gcut == wcut).all(axis=1)
        if top_p >= 1:
            assert same[live].all()
        assert same[live].sum() >= live.sum() - 1
        clear = live & same & (margin > 1e-5)
        assert np.array_equal(got[clear], want[clear])
