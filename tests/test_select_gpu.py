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


def _same_end(logits, T, min_p, top_k, top_p, got, want):
    """Whether the row's two ends are one. Ends that differ have to lie where the arithmetic leaves it open: weights come from two
    expf's (2 units apart), masses from 256 additions in a shard and one a shard, so relative to the mass each within
    b = (256 + shards) 2^-24 + 2^-22; of the two sets, one inside the other, all but the smaller one's last token weigh no more
    than the nucleus and the larger one more than it."""
    if (got == want).all():
        return True
    assert 0 < top_p < 1
    x = logits.astype(np.float64)
    live = np.flatnonzero(~np.isnan(logits) & (logits != -np.inf))
    order = live[np.lexsort((live, -x[live]))]                   # value descending, id ascending
    w = np.exp((x[order] - x[order[0]]) / T)
    n = len(order)
    if min_p > 0:
        n = int((x[order] >= min(np.float64(np.float32(x[order[0]] + T * np.log(min_p))), x[order[0]])).sum())
    if 0 < top_k < n:
        n = top_k
    mass = np.cumsum(w[:n])
    nucleus = top_p * mass[-1]
    bits = (logits[order] + np.float32(0)).view(np.uint32)
    key = np.where(bits >> 31 != 0, ~bits, bits | np.uint32(0x80000000))
    kept = [int(((key[:n] > e[0]) | ((key[:n] == e[0]) & (order[:n] <= e[1]))).sum()) for e in (got, want)]
    b = (256 + (len(logits) + 255) // 256) * 2.0 ** -24 + 2.0 ** -22
    a, z = min(kept), max(kept)
    # the end is the first token with which the mass passes the nucleus, give or take
    assert a >= 1 and mass[a - 1] >= nucleus * (1 - 2 * b) and (z < 2 or mass[z - 2] <= nucleus * (1 + 2 * b)), (kept, mass[a - 1] / nucleus, mass[z - 2] / nucleus)
    return False


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
        # A selection moves only where its test lies within the sums' roundings (margin, relative).
        same = np.array([not live[r] or _same_end(logits[r], T, min_p, top_k, top_p, gcut[r], wcut[r]) for r in range(rows)])
        clear = live & same & (margin > 1e-5)
        assert np.array_equal(got[clear], want[clear])


@pytest.mark.parametrize("vocab,policy", [(30000, (0.0, 0, 0.95)), (151936, (0.0, 0, 0.95)), (262144, (0.0, 0, 0.5)), (262144, (0.0, 90000, 1.0)),
                                          (262144, (0.0, 60000, 0.9))])
def test_ends_among_many_tokens(vocab, policy):
    """Distributions so broad that the end lies among tokens that weigh less than the sums' roundings, in bins that hold more of them
    than the list; one row with thirty values only, so that no division of a bin helps."""
    from splash_b200 import lib
    lib.init(0)
    l, o = lib.ops(), ol.bind_ops(ol.load())
    rows, (min_p, top_k, top_p) = 5, policy
    rng = np.random.default_rng(vocab)
    logits = (rng.standard_normal((rows, vocab)) * np.array([1.8, 1.8, 0.6, 0.05, 1.8])[:, None]).astype(np.float32)
    logits[1, rng.integers(0, vocab, 64)] = (6 + 3 * rng.standard_normal(64)).astype(np.float32)
    logits[4] = np.round(logits[4] * 4) / 4
    inputs, uniforms = rng.integers(0, vocab, rows).astype(np.uint32), rng.random(80).astype(np.float32)
    ld, idd, ud = (lib.DeviceBuffer.from_numpy(x) for x in (logits, inputs, uniforms))
    sd, cd, wd = lib.DeviceBuffer(rows * 4), lib.DeviceBuffer(rows * 8), lib.DeviceBuffer(int(l.sb_sample_workspace_bytes(rows, vocab)))
    a = lib.SbSampleArgs(ld.ptr, idd.ptr, ud.ptr, sd.ptr, wd.ptr, rows, vocab, vocab, 1.0, min_p, top_k, top_p, cd.ptr)
    lib.check(l.sb_sample_verify(None, ctypes.byref(a)))
    got, gcut = sd.to_numpy(np.uint32, (rows,)), cd.to_numpy(np.uint32, (rows, 2))
    want, margin, wcut = np.zeros(rows, np.uint32), np.zeros(rows, np.float64), np.zeros((rows, 2), np.uint32)
    o.so_sample_verify_filtered(P(logits), vocab, vocab, rows, P(inputs), 1.0, min_p, top_k, top_p, P(uniforms), P(want), P(margin), P(wcut))
    same = np.array([_same_end(logits[r], 1.0, min_p, top_k, top_p, gcut[r], wcut[r]) for r in range(rows)])
    if top_p >= 1:
        assert same.all()
    # (a draw from so many tokens lands within a unit of a prefix often enough: where it differs it lands next to the oracle's)
    for r in np.flatnonzero(same & (margin > 1e-5)):
        if got[r] != want[r]:
            w = np.exp(logits[r].astype(np.float64) - float(logits[r].max()))
            lo, hi = sorted((int(got[r]), int(want[r])))
            assert w[lo:hi].sum() <= 2.0 ** -12 * w.sum()


@pytest.mark.parametrize("temperature,vocab,sides", [(0.0, 20000, (2, 3)), (0.8, 200000, (15, 16))])
def test_the_two_kernels_select_alike(temperature, vocab, sides):
    """Either side of the counts of rows at which a launch changes kernels (greedy: above 32 rows; sampled without filters, a vocabulary
    that leaves one CTA a SM: from 256): the rows both launches hold get the same tokens, bit for bit."""
    from splash_b200 import lib
    lib.init(0)
    l = lib.ops()
    lanes = max(sides)
    rng = np.random.default_rng(lanes)
    base = (rng.standard_normal((16, vocab)) * 2).astype(np.float32)
    base[3] = np.round(base[3])
    logits = lib.DeviceBuffer(lanes * 16 * vocab * 4)
    for z in range(lanes):
        logits.upload(np.roll(base, 977 * z, axis=1), offset=z * base.nbytes)
    inputs = np.tile(base.argmax(axis=1), lanes).astype(np.uint32)
    idd, ud = lib.DeviceBuffer.from_numpy(inputs), lib.DeviceBuffer.from_numpy(rng.random((lanes, 80)).astype(np.float32))
    wd = lib.DeviceBuffer(int(l.sb_sample_workspace_bytes(lanes * 16, vocab)))
    got = []
    for n in sides:
        sd = lib.DeviceBuffer(lanes * 16 * 4)
        a = lib.SbSampleArgs(logits.ptr, idd.ptr, ud.ptr, sd.ptr, wd.ptr, 16, vocab, vocab, temperature, 0.0, 0, 1.0)
        a.lanes = n
        lib.check(l.sb_sample_verify(None, ctypes.byref(a)))
        got.append(sd.to_numpy(np.uint32, (n * 16,)))
    common = 16 * min(sides)
    assert np.array_equal(got[0][:common], got[1][:common])
    if temperature == 0.0:
        assert np.array_equal(got[1], np.concatenate([np.roll(base, 977 * z, axis=1).argmax(axis=1) for z in range(lanes)]))


@pytest.mark.parametrize("lanes,rows,vocab", [(1, 16, 3000), (2, 16, 50257), (3, 13, 3001), (9, 16, 200000), (64, 5, 2049)])
def test_policies_a_lane_equal_launches_of_one_policy(lanes, rows, vocab):
    """Greedy lanes among sampled ones (their rows take a CTA each where the launch has many): the tokens of a launch with the lane's
    policy for all."""
    from splash_b200 import lib
    lib.init(0)
    l = lib.ops()
    rng = np.random.default_rng(lanes * 100 + rows)
    base = (rng.standard_normal((16, vocab)) * 2).astype(np.float32)
    base[1, 7:19] = 30.0
    base[2] = np.nan
    logits = lib.DeviceBuffer(lanes * base.nbytes + 16)
    for z in range(lanes):
        logits.upload(np.roll(base, 977 * z, axis=1), offset=z * base.nbytes)
    policies = [(0.0, 0.0, 0, 1.0), (0.7, 0.0, 50, 0.95), (0.9, 0.02, 0, 1.0)]
    idd = lib.DeviceBuffer.from_numpy(rng.integers(0, vocab, (lanes, 16)).astype(np.uint32))
    ud = lib.DeviceBuffer.from_numpy(rng.random((lanes, 80)).astype(np.float32))
    wd = lib.DeviceBuffer(int(l.sb_sample_workspace_bytes(lanes * 16, vocab)))

    def select(policy, table=None):
        sd = lib.DeviceBuffer(lanes * 16 * 4)
        sd.fill(0)
        a = lib.SbSampleArgs(logits.ptr, idd.ptr, ud.ptr, sd.ptr, wd.ptr, rows, vocab, vocab, *policy)
        a.lanes = lanes if lanes > 1 else 0
        if table is not None:
            a.lane_policies = table.ptr
        lib.check(l.sb_sample_verify(None, ctypes.byref(a)))
        lib.stream_sync()
        assert lib.device_status() == 0
        return sd.to_numpy(np.uint32, (lanes, 16))[:, :rows]

    one = [select(p) for p in policies]
    for shift, kinds in ((0, 3), (1, 3), (0, 1)):
        which = [(z + shift) % kinds for z in range(lanes)]
        table = lib.DeviceBuffer.from_numpy(np.frombuffer(bytes((lib.SbLanePolicy * lanes)(*[lib.SbLanePolicy(*policies[k]) for k in which])), np.uint8).copy())
        got = select(policies[1], table)
        for z in range(lanes):
            assert np.array_equal(got[z], one[which[z]][z]), (z, which[z])
