"""The verify step's work as a program that serves requests has it done, case by case: whole steps of a target, its layers
(feed-forward block, attention, Gated DeltaNet, MoE block) and the selection of the next tokens, each through the calls
of include/splash_b200.h that such a program makes.

A case is a dict of plain values. `listed()` names the sizes that are always looked at, `draw(rng)` gives more of the same
ranges, `prepare` makes what the caller holds before the call, `run` makes one pass, `exact` states the same results in
64 bits with plain torch."""
import ctypes
import math

import numpy as np
import torch

from splash_b200 import lib, target

GIB = 1 << 30
FMT = {"q4k": lib.FMT_Q4K, "q6k": lib.FMT_Q6K, "q80": lib.FMT_Q80, "nvfp4": lib.FMT_NVFP4}
BLOCK = {"q4k": (256, 144), "q6k": (256, 210), "q80": (32, 34), "nvfp4": (256, 148)}  # weights a block, bytes a block
GDN_DIM = 128
ROW_SLOTS = 16  # row slots of a lane


def listed():
    ffn27 = dict(kind="ffn", hidden=5120, inter=17408, gate_up="q4k", down="q6k")
    att27 = dict(kind="attention", q_heads=24, kv_heads=4, head_dim=256, pairs=32, page_tokens=256, half_scales=True)
    gdn27 = dict(kind="gdn", key_heads=16, value_heads=48, hidden=5120, tiled=True)
    moe35 = dict(kind="moe", hidden=2048, inter=512, experts=256, top_k=8)
    return [
        # A small hybrid model's whole step: what a step costs when no kernel has much to do (launches, hand-offs).
        dict(name="step_small", kind="step", model="tiny", layers=4, lanes=1, rows=16, context=2048, temperature=0.0),
        # The headline workload: one request on the 27B shape, 32K tokens of context, a block of 16 draft tokens.
        dict(name="step_27b_32k", kind="step", model="27b", layers=64, lanes=1, rows=16, context=32768, temperature=0.0),
        # One 27B feed-forward block (norm, gate/up, down, residual) for one request: the projections are most of a step.
        dict(ffn27, name="ffn_one_lane", rows=16),
        # The same for eight requests stepped together.
        dict(ffn27, name="ffn_eight_lanes", rows=128),
        # A small model's block, Q8_0, and a short draft: odd row count, narrow matrices.
        dict(name="ffn_short_block_q80", kind="ffn", hidden=1024, inter=2816, gate_up="q80", down="q80", rows=5),
        # One attention layer of the 27B shape at 32K (store the block's keys and values, then attend).
        dict(att27, name="attention_32k", lanes=1, rows=16, context=32768, spread=0, tree=False),
        # Eight requests of different lengths around 8K, every block a draft tree.
        dict(att27, name="attention_eight_lanes_trees", lanes=8, rows=13, context=8111, spread=3000, tree=True),
        # One Gated-DeltaNet layer of the 27B shape, six rows of the last step to fold in.
        dict(gdn27, name="gdn_one_lane", lanes=1, rows=16, pending=6, tree=False),
        # Eight requests.
        dict(gdn27, name="gdn_eight_lanes", lanes=8, rows=16, pending=6, tree=False),
        # One MoE block of the 35B-A3B shape (routing and experts) for one request, and for 32 requests.
        dict(moe35, name="moe_one_lane", rows=16),
        dict(moe35, name="moe_32_lanes", rows=512),
        # Next tokens of eight requests sampled at temperature 0.7 with top-k and top-p, acceptance of the drafts included.
        dict(name="select_eight_lanes", kind="select", lanes=8, rows=16, vocab=151936, temperature=0.7, min_p=0.0, top_k=50, top_p=0.95),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def draw(rng):
    kind = rng.choice(["step", "ffn", "ffn", "attention", "attention", "gdn", "gdn", "moe", "moe", "select", "select"])
    if kind == "step":
        return dict(kind="step", model=rng.choice(["tiny", "27b"]), layers=4 * rng.randint(1, 4), lanes=rng.choice([1, 1, 2, 3, 8]), rows=rng.randint(1, 16),
                    context=_log_int(rng, 100, 20000), temperature=rng.choice([0.0, 0.0, 0.7]))
    if kind == "ffn":
        lanes = rng.choice([1, 1, 2, 4, 8, 32])
        fmt = rng.choice(["q4k", "q4k", "q6k", "q80", "nvfp4"])
        return dict(kind="ffn", hidden=256 * _log_int(rng, 4, 20), inter=256 * _log_int(rng, 8, 68), gate_up=fmt, down=fmt if fmt == "nvfp4" else rng.choice(["q4k", "q6k", "q80"]),
                    rows=rng.randint(1, 16) if lanes == 1 else 16 * lanes)
    if kind == "attention":
        lanes = rng.choice([1, 1, 2, 3, 8])
        context = _log_int(rng, 40, 131072 if lanes == 1 else 65536 // lanes)
        kv = rng.choice([2, 4])
        return dict(kind="attention", q_heads=kv * rng.choice([1, 4, 6, 8]), kv_heads=kv, head_dim=rng.choice([128, 256, 256]), pairs=32, page_tokens=rng.choice([64, 256]),
                    half_scales=rng.random() < 0.7, lanes=lanes, rows=rng.randint(1, 16), context=context, spread=rng.randint(0, context - 1) if lanes > 1 else 0,
                    tree=rng.random() < 0.4)
    if kind == "gdn":
        kh = rng.choice([4, 8, 16])
        return dict(kind="gdn", key_heads=kh, value_heads=kh * rng.choice([1, 2, 3]), hidden=256 * _log_int(rng, 4, 20), lanes=rng.choice([1, 1, 2, 3, 8, 32]),
                    tiled=rng.random() < 0.5, rows=rng.randint(1, 16), pending=rng.randint(0, 16), tree=rng.random() < 0.4)
    if kind == "moe":
        lanes = rng.choice([1, 1, 2, 8, 32])
        return dict(kind="moe", hidden=256 * _log_int(rng, 4, 8), inter=256 * rng.randint(1, 3), experts=rng.choice([64, 128, 256]), top_k=rng.randint(2, 8),
                    rows=rng.randint(1, 16) if lanes == 1 else 16 * lanes)
    filters = rng.choice([(0.0, 0, 1.0), (0.05, 0, 1.0), (0.0, 50, 0.95), (0.02, 200, 0.9), (0.0, 0, 0.95)])
    return dict(kind="select", lanes=rng.choice([1, 1, 2, 8, 32]), rows=rng.randint(1, 16), vocab=_log_int(rng, 30000, 250000), temperature=rng.choice([0.0, 0.6, 0.7, 1.0]),
                min_p=filters[0], top_k=filters[1], top_p=filters[2])


# ---- shared pieces ----

def _device():
    d = torch.device("cuda", torch.cuda.current_device())
    torch.empty(1, device=d)
    lib.init(d.index)
    return d


def _generator(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _bf16(g, shape, scale=1.0):
    return (torch.randn(shape, generator=g, device=g.device) * scale).to(torch.bfloat16)


def _uniform(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device=g.device) * (hi - lo) + lo


def _tree_masks(rows, seed, lane):
    """Ancestor masks and parents of a draft tree: a row's parent is one of the three rows before it."""
    rng = torch.Generator().manual_seed(int(seed) * 131 + lane)
    anc, parent = [1], [0]
    for r in range(1, rows):
        p = max(0, r - 1 - int(torch.randint(0, 3, (1,), generator=rng)))
        anc.append(anc[p] | (1 << r))
        parent.append(p)
    return anc, parent


def _tree_tensor(lanes, rows, seed, tree, device):
    out = torch.zeros((lanes, ROW_SLOTS, 2), dtype=torch.int64)
    for l in range(lanes):
        anc, parent = _tree_masks(rows, seed, l) if tree else ([(2 << r) - 1 for r in range(rows)], [max(r - 1, 0) for r in range(rows)])
        for r in range(rows):
            out[l, r, 0] = anc[r]
            out[l, r, 1] = parent[r] | ((bin(anc[r]).count("1") - 1) << 16)
    return out.to(torch.int32).to(device)


class _DeviceArray:
    """A library buffer as torch sees it (no copy); holds its owner."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr, data=(ptr, False), strides=None, version=3)


# ---- quantized rows ----

def _native_rows(g, fmt, n, k):
    """n native rows of k weights with scales of the size trained files hold (values around 0.02), other bytes uniform."""
    elements, size = BLOCK[fmt]
    nb = k // elements
    blk = torch.randint(0, 256, (n, nb, size), generator=g, device=g.device, dtype=torch.uint8)
    half = lambda lo, hi: _uniform(g, (n, nb), lo, hi).to(torch.float16).view(torch.uint8).reshape(n, nb, 2)
    if fmt == "q4k":
        blk[..., 0:2], blk[..., 2:4] = half(5e-5, 4e-4), half(3e-4, 3e-3)
    elif fmt == "q6k":
        blk[..., 192:208] = torch.randint(-64, 64, (n, nb, 16), generator=g, device=g.device, dtype=torch.int8).view(torch.uint8)
        blk[..., 208:210] = half(2e-5, 4e-5)
    elif fmt == "q80":
        blk[..., 0:2] = half(1e-4, 6e-4)
    else:
        blk[..., 0:16] = torch.randint(0x28, 0x40, (n, nb, 16), generator=g, device=g.device, dtype=torch.uint8)
        blk[..., 16:20] = torch.full((n, nb), 5e-3, device=g.device).view(torch.uint8).reshape(n, nb, 4)
    return blk.reshape(n, nb * size)


def _half64(b):
    return b.contiguous().view(torch.float16).squeeze(-1).double()


def _dequant64(fmt, rows, k):
    elements, size = BLOCK[fmt]
    n = rows.shape[0]
    b = rows.reshape(n, k // elements, size)
    nb = b.shape[1]
    if fmt == "q80":
        return (_half64(b[..., 0:2]).unsqueeze(-1) * b[..., 2:].contiguous().view(torch.int8).double()).reshape(n, k)
    if fmt == "q4k":
        d, dmin, s = _half64(b[..., 0:2]), _half64(b[..., 2:4]), b[..., 4:16].to(torch.int32)
        sc = torch.cat([s[..., 0:4] & 63, (s[..., 8:12] & 15) | ((s[..., 0:4] >> 6) << 4)], -1).double()
        mn = torch.cat([s[..., 4:8] & 63, (s[..., 8:12] >> 4) | ((s[..., 4:8] >> 6) << 4)], -1).double()
        q = b[..., 16:].reshape(n, nb, 4, 1, 32).expand(n, nb, 4, 2, 32).to(torch.int32)
        q = (q >> torch.tensor([0, 4], device=q.device).reshape(1, 1, 1, 2, 1)) & 15
        q = q.reshape(n, nb, 8, 32).double()
        return ((d.unsqueeze(-1) * sc).unsqueeze(-1) * q - (dmin.unsqueeze(-1) * mn).unsqueeze(-1)).reshape(n, k)
    if fmt == "q6k":
        d, sc = _half64(b[..., 208:210]), b[..., 192:208].contiguous().view(torch.int8).double()
        ql, qh = b[..., 0:128].to(torch.int32).reshape(n, nb, 2, 2, 32), b[..., 128:192].to(torch.int32).reshape(n, nb, 2, 32)
        parts = []
        for r in range(4):
            lo = (ql[:, :, :, r & 1] >> (4 * (r >> 1))) & 15
            parts.append(lo | (((qh >> (2 * r)) & 3) << 4))
        q = torch.stack(parts, 3).double() - 32.0  # [n, nb, 2, 4, 32]
        return (d.reshape(n, nb, 1, 1, 1, 1) * sc.reshape(n, nb, 2, 4, 2, 1) * q.reshape(n, nb, 2, 4, 2, 16)).reshape(n, k)
    e4m3 = b[..., 0:16].contiguous().view(torch.float8_e4m3fn).to(torch.float64)
    g = b[..., 16:20].contiguous().view(torch.float32).squeeze(-1).double()
    table = torch.tensor([0, 1, 2, 3, 4, 6, 8, 12, 0, -1, -2, -3, -4, -6, -8, -12], dtype=torch.float64, device=b.device)
    codes = b[..., 20:].to(torch.int64).unsqueeze(-1)
    codes = torch.cat([codes & 15, codes >> 4], -1).reshape(n, nb, 16, 16)
    return (table[codes] * (e4m3 * g.unsqueeze(-1) * 0.5).unsqueeze(-1)).reshape(n, k)


def _matmul64(x, fmt, rows, k, chunk=4096):
    return torch.cat([x @ _dequant64(fmt, rows[i:i + chunk], k).T for i in range(0, rows.shape[0], chunk)], -1)


def _rms64(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w


# ---- feed-forward block: hidden + down(silu(gate(norm)) * up(norm)), and the conversion the next projection reads ----

def _ffn_inputs(case, seed, device):
    g = _generator(seed, device)
    H, I, M = case["hidden"], case["inter"], case["rows"]
    return dict(x=_bf16(g, (max(ROW_SLOTS, M), H)), norm=_uniform(g, (H,), 0.7, 1.3), next_norm=_uniform(g, (H,), 0.7, 1.3),
                gate=_native_rows(g, case["gate_up"], I, H), up=_native_rows(g, case["gate_up"], I, H), down=_native_rows(g, case["down"], H, I))


def _wide(case):
    return case["rows"] > ROW_SLOTS or "nvfp4" in (case["gate_up"], case["down"])


def _image(l, fmt, rows, n, k):
    if fmt == "q4k":
        return rows, 0
    l.sb_linear_wide_image_bytes.restype = ctypes.c_uint64
    out = torch.empty(int(l.sb_linear_wide_image_bytes(FMT[fmt], n, k)), dtype=torch.uint8, device=rows.device)
    lib.check(l.sb_linear_wide_image(_stream(), FMT[fmt], rows.data_ptr(), n, k, out.data_ptr()))
    return out, lib.LINEAR_WIDE_IMAGE


def _prepare_ffn(case, seed):
    d = _device()
    l = lib.ops()
    H, I, M = case["hidden"], case["inter"], case["rows"]
    s = _ffn_inputs(case, seed, d)
    slots = max(ROW_SLOTS, M)
    wide = _wide(case)
    s["act"] = torch.zeros((slots, I), dtype=torch.bfloat16, device=d)
    s["out"] = torch.zeros((slots, H), dtype=torch.bfloat16, device=d)
    u, p = ctypes.c_uint32, ctypes.c_void_p
    if wide:
        l.sb_linear_wide_splits.argtypes = [u, u]
        l.sb_linear_wide_splits.restype = u
        l.sb_linear_wide_prepare_sum.argtypes = [p, p, u, u, p, u, p, u, u, u, p, p, u]
        l.sb_linear_wide_prepared_bytes.restype = ctypes.c_uint64
        s["slices"] = int(l.sb_linear_wide_splits(H, I))
        s["prep"] = [torch.empty(int(l.sb_linear_wide_prepared_bytes(M, k)), dtype=torch.uint8, device=d) for k in (H, I, H)]
        for key, fmt, n, k in (("gate", case["gate_up"], I, H), ("up", case["gate_up"], I, H), ("down", case["down"], H, I)):
            s[key], s[key + "_flags"] = _image(l, fmt, s[key], n, k)
    else:
        plan = lib.SbLinearPlan()
        lib.check(l.sb_linear_plan(FMT[case["down"]], H, I, M, lib.EP_PARTIALS, ctypes.byref(plan)))
        s["slices"] = int(plan.slices)
        s["prep"] = [torch.empty(int(l.sb_linear_prepared_bytes(k)), dtype=torch.uint8, device=d) for k in (H, I, H)]
    s["partials"] = torch.empty((s["slices"], slots, H), dtype=torch.float32, device=d)
    s["case"], s["wide"], s["lib"] = case, wide, l
    torch.cuda.current_stream().synchronize()
    return s


def _run_ffn(s):
    case, l, st = s["case"], s["lib"], _stream()
    H, I, M = case["hidden"], case["inter"], case["rows"]
    ptr = lambda k: s[k].data_ptr()
    prep = [t.data_ptr() for t in s["prep"]]
    gf, df = FMT[case["gate_up"]], FMT[case["down"]]
    if s["wide"]:
        lib.check(l.sb_linear_wide_prepare(st, ptr("x"), M, H, H, ptr("norm"), prep[0], lib.LINEAR_PDL))
        a = lib.SbLinearArgs(ptr("gate"), ptr("up"), None, prep[0], None, ptr("act"), None, gf, I, H, M, H, 0, I, lib.EP_GATE_UP, 0, lib.LINEAR_PDL | s["gate_flags"])
        lib.check(l.sb_linear(st, ctypes.byref(a)))
        lib.check(l.sb_linear_wide_prepare(st, ptr("act"), M, I, I, None, prep[1], lib.LINEAR_PDL))
        a = lib.SbLinearArgs(ptr("down"), None, None, prep[1], None, ptr("partials"), None, df, H, I, M, I, 0, H, lib.EP_PARTIALS, 1, lib.LINEAR_PDL | s["down_flags"])
        lib.check(l.sb_linear(st, ctypes.byref(a)))
        lib.check(l.sb_linear_wide_prepare_sum(st, ptr("partials"), s["slices"], H, ptr("x"), H, ptr("out"), H, M, H, ptr("next_norm"), prep[2], lib.LINEAR_PDL))
    else:
        lib.check(l.sb_linear_prepare(st, ptr("x"), M, H, H, ptr("norm"), gf, prep[0], None, lib.LINEAR_PDL))
        a = lib.SbLinearArgs(ptr("gate"), ptr("up"), None, prep[0], None, ptr("act"), None, gf, I, H, M, H, 0, I, lib.EP_GATE_UP, 0, lib.LINEAR_PDL)
        lib.check(l.sb_linear(st, ctypes.byref(a)))
        lib.check(l.sb_linear_prepare(st, ptr("act"), M, I, I, None, df, prep[1], None, lib.LINEAR_PDL))
        a = lib.SbLinearArgs(ptr("down"), None, None, prep[1], None, ptr("partials"), None, df, H, I, M, I, 0, H, lib.EP_PARTIALS, 1, lib.LINEAR_PDL)
        lib.check(l.sb_linear(st, ctypes.byref(a)))
        lib.check(l.sb_linear_prepare_sum(st, ptr("partials"), s["slices"], H, ptr("x"), H, ptr("out"), H, M, H, ptr("next_norm"), gf, prep[2], None, lib.LINEAR_PDL))
    return {"act": s["act"][:M], "hidden": s["out"][:M]}  # (the slots past the block's rows hold nothing)


def _exact_ffn(case, seed):
    s = _ffn_inputs(case, seed, _device())
    x = s["x"][:case["rows"]].double()
    n = _rms64(x, s["norm"].double())
    gate, up = (_matmul64(n, case["gate_up"], s[k], case["hidden"]) for k in ("gate", "up"))
    act = up * gate * torch.sigmoid(gate)
    return {"act": act, "hidden": x + _matmul64(act, case["down"], s["down"], case["inter"])}


def _work_ffn(case):
    H, I, M = case["hidden"], case["inter"], case["rows"]
    per = lambda f: BLOCK[f][1] / BLOCK[f][0]
    return {"bytes": int(2 * I * H * per(case["gate_up"]) + H * I * per(case["down"]) + 2 * M * (2 * H + I) + 8 * H), "flops": 6 * M * H * I}


# ---- attention layer: q/k norm, RoPE, INT8 store of the block's rows, attention over the pages, output gate ----

def _attention_positions(case, seed):
    rng = torch.Generator().manual_seed(int(seed) + 17)
    return [case["context"]] + [case["context"] - int(torch.randint(0, case["spread"] + 1, (1,), generator=rng)) for _ in range(case["lanes"] - 1)]


def _attention_inputs(case, seed, device):
    g = _generator(seed, device)
    L, Q, K, D, P = case["lanes"], case["q_heads"], case["kv_heads"], case["head_dim"], case["page_tokens"]
    positions = _attention_positions(case, seed)
    pages = (case["context"] + ROW_SLOTS + P - 1) // P
    pool = L * pages
    scale_type = torch.float16 if case["half_scales"] else torch.float32
    tree = _tree_tensor(L, case["rows"], seed, case["tree"], device)
    depth = (tree[..., 1] >> 16).float()
    angles = (torch.tensor(positions, device=device, dtype=torch.float32).reshape(L, 1) + depth).reshape(L * ROW_SLOTS, 1) * (
        1e7 ** (-torch.arange(case["pairs"], device=device, dtype=torch.float64) / case["pairs"])).float().reshape(1, -1)
    return dict(
        qkv=_bf16(g, (L * ROW_SLOTS, Q * 2 * D + 2 * K * D)), q_norm=_uniform(g, (D,), 0.8, 1.4), k_norm=_uniform(g, (D,), 0.8, 1.4),
        k=torch.randint(-127, 128, (pool, K, P, D), generator=g, device=device, dtype=torch.int8),
        v=torch.randint(-127, 128, (pool, K, P, D), generator=g, device=device, dtype=torch.int8),
        ks=_uniform(g, (pool, K, P), 0.008, 0.03).to(scale_type), vs=_uniform(g, (pool, K, P), 0.008, 0.03).to(scale_type),
        table=torch.randperm(pool, generator=g, device=device).to(torch.int32).reshape(L, pages), tree=tree,
        cos=torch.cos(angles).contiguous(), sin=torch.sin(angles).contiguous(), positions=torch.tensor(positions, dtype=torch.int32, device=device))


def _prepare_attention(case, seed):
    d = _device()
    l = lib.ops()
    lib.check(l.sb_set_attention_kernel(0))
    s = _attention_inputs(case, seed, d)
    L, Q, K, D = case["lanes"], case["q_heads"], case["kv_heads"], case["head_dim"]
    s["queries"] = torch.zeros((L * ROW_SLOTS, Q, D), dtype=torch.bfloat16, device=d)
    s["out"] = torch.zeros((L * ROW_SLOTS, Q * D), dtype=torch.bfloat16, device=d)
    p = lambda k: s[k].data_ptr()
    cache = lib.SbKvLayer(p("k"), p("v"), p("ks"), p("vs"), K, D, case["page_tokens"], int(case["half_scales"]))
    stride, lanes, pages = s["qkv"].shape[1], L if L > 1 else 0, s["table"].shape[1]
    s["store"] = lib.SbAttnStoreArgs(p("qkv"), p("q_norm"), p("k_norm"), p("cos"), p("sin"), p("table"), p("queries"), cache, p("positions"),
                                     case["rows"], Q, 1, case["pairs"], stride, case["context"], lanes, pages)
    s["attend"] = lib.SbAttnArgs(p("queries"), p("qkv"), p("table"), p("tree") if case["tree"] else None, p("out"), cache, p("positions"),
                                 case["rows"], Q, 1, stride, Q * D, case["context"], lanes, pages)
    s["case"], s["lib"] = case, l
    torch.cuda.current_stream().synchronize()
    return s


def _lane_rows(t, case):
    """The block's rows of every lane (the row slots past them hold nothing)."""
    return t.reshape((case["lanes"], ROW_SLOTS) + t.shape[1:])[:, :case["rows"]]


def _run_attention(s):
    l, st = s["lib"], _stream()
    lib.check(l.sb_attn_store(st, ctypes.byref(s["store"])))
    lib.check(l.sb_attn_verify(st, ctypes.byref(s["attend"])))
    return {"out": _lane_rows(s["out"], s["case"]), "queries": _lane_rows(s["queries"], s["case"]), "k": s["k"], "v": s["v"], "k_scale": s["ks"], "v_scale": s["vs"]}


def _exact_attention(case, seed):
    s = _attention_inputs(case, seed, _device())
    L, Q, K, D, P, R = case["lanes"], case["q_heads"], case["kv_heads"], case["head_dim"], case["page_tokens"], case["rows"]
    qkv = _lane_rows(s["qkv"], case).double()
    cos, sin = (_lane_rows(s[k], case).double().unsqueeze(2) for k in ("cos", "sin"))

    def norm_rope(x, w):
        x = _rms64(x, w.double())
        a, b = x[..., :case["pairs"]], x[..., case["pairs"]:2 * case["pairs"]]
        return torch.cat([a * cos - b * sin, b * cos + a * sin, x[..., 2 * case["pairs"]:]], -1)

    qg = qkv[..., :Q * 2 * D].reshape(L, R, Q, 2 * D)
    gate = qg[..., D:]
    q = norm_rope(qg[..., :D], s["q_norm"])
    k_new = norm_rope(qkv[..., Q * 2 * D:Q * 2 * D + K * D].reshape(L, R, K, D), s["k_norm"])
    v_new = qkv[..., Q * 2 * D + K * D:].reshape(L, R, K, D)
    out = torch.empty((L, R, Q * D), dtype=torch.float64, device=qkv.device)
    for i in range(L):
        pos, pages = int(s["positions"][i]), s["table"][i].long()
        flat = lambda c, sc: (s[c][pages].double() * s[sc][pages].double().unsqueeze(-1)).transpose(0, 1).reshape(K, -1, D)[:, :pos + R].clone()
        for h in range(K):
            kk, vv = ((s[c][pages, h].double() * s[sc][pages, h].double().unsqueeze(-1)).reshape(-1, D)[:pos + R] for c, sc in (("k", "ks"), ("v", "vs")))
            kk[pos:], vv[pos:] = k_new[i, :, h], v_new[i, :, h]  # (the stored rows' codes differ from these by their quantization)
            G = Q // K
            qq = q[i, :, h * G:(h + 1) * G].reshape(R * G, D)
            score = (qq @ kk.T) / math.sqrt(D)
            seen = (s["tree"][i, :R, 0].long().reshape(R, 1) >> torch.arange(R, device=qkv.device).reshape(1, R)) & 1
            score.reshape(R, G, -1)[:, :, pos:].masked_fill_((seen == 0).unsqueeze(1), float("-inf"))
            o = (torch.softmax(score, -1) @ vv).reshape(R, G, D)
            out[i, :, h * G * D:(h + 1) * G * D] = (o * torch.sigmoid(gate[i, :, h * G:(h + 1) * G])).reshape(R, G * D)
    return {"out": out, "queries": q, "k": None, "v": None, "k_scale": None, "v_scale": None}


def _work_attention(case):
    L, Q, K, D, R = case["lanes"], case["q_heads"], case["kv_heads"], case["head_dim"], case["rows"]
    tokens = case["context"] + (L - 1) * (case["context"] - case["spread"] // 2)  # (the lanes' positions lie evenly below the context)
    per_token = 2 * K * (D + (2 if case["half_scales"] else 4))
    rows = L * R * 2 * (Q * 2 * D + 2 * K * D + 2 * Q * D)
    return {"bytes": int(tokens * per_token + rows + L * R * per_token), "flops": int(4 * tokens * R * Q * D)}


# ---- Gated-DeltaNet layer: alpha / beta projection, fold of the last step's accepted rows, conv, norms, scan, gated norm ----

def _gdn_inputs(case, seed, device):
    g = _generator(seed, device)
    L, KH, VH, H, R = case["lanes"], case["key_heads"], case["value_heads"], case["hidden"], ROW_SLOTS
    KW, VW = KH * GDN_DIM, VH * GDN_DIM
    C = 2 * KW + VW
    keys = torch.nn.functional.normalize(torch.randn((L * R, KH, GDN_DIM), generator=g, device=device), dim=-1).reshape(L * R, KW)
    masks = []
    for i in range(L):  # the accepted path's rows in the last step's tape: its first rows, or a path down its tree
        if case["tree"] and case["pending"]:
            masks.append(_tree_masks(case["pending"], seed + 1, i)[0][-1])
        else:
            masks.append((1 << case["pending"]) - 1)
    return dict(
        qkvz=_bf16(g, (L * R, C + VW)), x=_bf16(g, (L * R, H)), gates=torch.randn((2 * VH, H), generator=g, device=device) / math.sqrt(H), conv_w=_bf16(g, (C, 4), 0.4),
        a_scale=-torch.exp(_uniform(g, (VH,), -3.0, 0.5)), dt_bias=_bf16(g, (VH,), 0.5), norm=_uniform(g, (GDN_DIM,), 0.7, 1.3), conv_in=_bf16(g, (L, 3, C)),
        state_in=torch.randn((L, VH, GDN_DIM, GDN_DIM), generator=g, device=device) * 0.05,
        p_inputs=_bf16(g, (L * R, C)), p_k=keys.to(torch.bfloat16), p_v=_bf16(g, (L * R, VW), 0.5), p_beta=_uniform(g, (L * R, VH), 0.1, 0.9).to(torch.bfloat16),
        p_decay=_uniform(g, (L * R, VH), 0.5, 1.0), tree=_tree_tensor(L, case["rows"], seed, case["tree"], device),
        pending=torch.tensor(masks if case["tree"] else [case["pending"]] * L, dtype=torch.int32, device=device), masks=masks)


def _prepare_gdn(case, seed):
    d = _device()
    l = lib.ops()
    s = _gdn_inputs(case, seed, d)
    L, KH, VH, R = case["lanes"], case["key_heads"], case["value_heads"], ROW_SLOTS
    KW, VW = KH * GDN_DIM, VH * GDN_DIM
    C = 2 * KW + VW
    bf = lambda *shape: torch.zeros(shape, dtype=torch.bfloat16, device=d)
    s.update(conv_out=bf(L, 3, C), state_out=torch.zeros_like(s["state_in"]), hidden=bf(L * R, VW), t_inputs=bf(L * R, C), t_k=bf(L * R, KW), t_v=bf(L * R, VW),
             t_beta=bf(L * R, VH), t_decay=torch.zeros((L * R, VH), device=d))
    p = lambda k: s[k].data_ptr()
    tape = lambda t: lib.SbGdnTape(p(t + "inputs"), p(t + "k"), p(t + "v"), p(t + "beta"), p(t + "decay"))
    a = lib.SbGdnArgs()
    a.qkvz, a.conv_w, a.a_scale, a.dt_bias, a.norm_w = p("qkvz"), p("conv_w"), p("a_scale"), p("dt_bias"), p("norm")
    a.conv_state_in, a.conv_state_out, a.state_in, a.state_out = p("conv_in"), p("conv_out"), p("state_in"), p("state_out")
    a.pending, a.step, a.hidden = tape("p_"), tape("t_"), p("hidden")
    a.rows, a.key_heads, a.value_heads, a.qkvz_stride, a.ab_stride, a.hidden_stride, a.tiled = case["rows"], KH, VH, C + VW, VH, VW, int(case["tiled"])
    a.gate_weight, a.gate_input, a.gate_k, a.gate_input_stride = p("gates"), p("x"), case["hidden"], case["hidden"]
    if case["tree"]:
        a.tree, a.pending_path_dev = p("tree"), p("pending")
    else:
        a.pending_rows_dev = p("pending")
    a.lanes = L if L > 1 else 0
    s["args"], s["case"], s["lib"] = a, case, l
    torch.cuda.current_stream().synchronize()
    return s


def _run_gdn(s):
    lib.check(s["lib"].sb_gdn_verify(_stream(), ctypes.byref(s["args"])))
    out = {k: _lane_rows(s[k], s["case"]) for k in ("hidden", "t_inputs", "t_k", "t_v", "t_beta", "t_decay")}
    out["state"], out["conv_state"] = s["state_out"], s["conv_out"]
    return out


def _exact_gdn(case, seed):
    s = _gdn_inputs(case, seed, _device())
    L, KH, VH, R, D = case["lanes"], case["key_heads"], case["value_heads"], case["rows"], GDN_DIM
    KW, VW, dev = KH * D, VH * D, s["qkvz"].device
    C = 2 * KW + VW
    lanes = lambda k: s[k].double().reshape((L, ROW_SLOTS) + s[k].shape[1:])
    qkvz = lanes("qkvz")[:, :R]
    inputs, z = qkvz[..., :C], qkvz[..., C:].reshape(L, R, VH, D)
    pin, pk, pv, pb, pd = (lanes("p_" + k) for k in ("inputs", "k", "v", "beta", "decay"))
    head = lambda t, n: t.reshape(t.shape[:-1] + (n, D))
    per_key = VH // KH
    ab = s["x"].double().reshape(L, ROW_SLOTS, -1)[:, :R] @ s["gates"].double().T
    beta = torch.sigmoid(ab[..., :VH])
    decay = torch.exp(s["a_scale"].double() * torch.nn.functional.softplus(ab[..., VH:] + s["dt_bias"].double()))
    conv_out, state_out = torch.empty((L, 3, C), dtype=torch.float64, device=dev), s["state_in"].double().clone()
    hidden = torch.empty((L, R, VW), dtype=torch.float64, device=dev)
    tk, tv = torch.empty((L, R, KW), dtype=torch.float64, device=dev), torch.empty((L, R, VW), dtype=torch.float64, device=dev)

    def advance(S, key, val, d, b):  # S [VH, D, D], key [VH, D], val [VH, D]
        S = S * d.reshape(VH, 1, 1)
        delta = (val - (S @ key.unsqueeze(-1)).squeeze(-1)) * b.unsqueeze(-1)
        return S + delta.unsqueeze(-1) * key.unsqueeze(1)

    for i in range(L):
        path = [r for r in range(ROW_SLOTS) if s["masks"][i] >> r & 1]
        hist = torch.cat([s["conv_in"][i].double(), pin[i][path]])[-3:]
        conv_out[i] = hist
        S = state_out[i]
        for r in path:
            S = advance(S, head(pk[i, r], KH).repeat_interleave(per_key, 0), head(pv[i, r], VH), pd[i, r], pb[i, r])
        state_out[i] = S
        states, taps = [], s["conv_w"].double()
        for r in range(R):
            anc = int(s["tree"][i, r, 0])
            mine = [t for t in range(r + 1) if anc >> t & 1]
            window = torch.cat([hist, inputs[i][mine]])[-4:]
            c = (window * taps.T).sum(0)
            c = c * torch.sigmoid(c)
            n = lambda x: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6)
            q, k, v = n(head(c[:KW], KH)) * 0.0078125, n(head(c[KW:2 * KW], KH)) * D ** -0.5, head(c[2 * KW:], VH)
            tk[i, r], tv[i, r] = k.reshape(-1), v.reshape(-1)
            T = advance(states[mine[-2]] if len(mine) > 1 else S, k.repeat_interleave(per_key, 0), v, decay[i, r], beta[i, r])
            states.append(T)
            o = (T @ q.repeat_interleave(per_key, 0).unsqueeze(-1)).squeeze(-1)
            o = n(o) * s["norm"].double() * z[i, r] * torch.sigmoid(z[i, r])
            if case["tiled"]:  # value head (key head, index) stands at index * key heads + key head
                o = o.reshape(KH, per_key, D).transpose(0, 1)
            hidden[i, r] = o.reshape(-1)
    return {"hidden": hidden, "t_inputs": inputs, "t_k": tk, "t_v": tv, "t_beta": beta, "t_decay": decay, "state": state_out, "conv_state": conv_out}


def _work_gdn(case):
    L, KH, VH, H, R, F = case["lanes"], case["key_heads"], case["value_heads"], case["hidden"], case["rows"], case["pending"]
    KW, VW = KH * GDN_DIM, VH * GDN_DIM
    C = 2 * KW + VW
    state = VH * GDN_DIM * GDN_DIM
    rows = R * 2 * (C + VW + H + VW + C + KW + VW) + F * 2 * (KW + VW) + 6 * R * VH
    return {"bytes": int(L * (8 * state + rows + 12 * C) + 8 * VH * H + 8 * C), "flops": int(L * (state * (4 * F + 6 * R) + 4 * R * VH * H))}


# ---- MoE block: routing from given router logits, the routed experts and the shared one, back onto the residual ----

def _moe_inputs(case, seed, device):
    g = _generator(seed, device)
    H, I, E, M = case["hidden"], case["inter"], case["experts"] + 1, case["rows"]
    return dict(x=_bf16(g, (M, H)), residual=_bf16(g, (M, H)), scores=torch.randn((M, case["experts"]), generator=g, device=device),
                shared_gate=torch.randn((H,), generator=g, device=device) * 0.05, gate=_native_rows(g, "q4k", E * I, H), up=_native_rows(g, "q4k", E * I, H),
                down=_native_rows(g, "q4k", E * H, I))


def _prepare_moe(case, seed):
    d = _device()
    l = lib.ops()
    s = _moe_inputs(case, seed, d)
    M, E, K, H, I = case["rows"], case["experts"], case["top_k"], case["hidden"], case["inter"]
    s["selected"] = torch.zeros((M, K + 1), dtype=torch.int32, device=d)
    s["weights"] = torch.zeros((M, K + 1), dtype=torch.float32, device=d)
    s["scratch"] = torch.empty(int(l.sb_moe_scratch_bytes(M, K + 1, H, I)), dtype=torch.uint8, device=d)
    s["out"] = torch.zeros((M, H), dtype=torch.bfloat16, device=d)
    p = lambda k: s[k].data_ptr()
    s["route"] = lib.SbMoeRouteArgs(p("scores"), p("x"), p("shared_gate"), p("selected"), p("weights"), M, E, E, K, H, 0)
    s["experts"] = lib.SbMoeExpertArgs(p("x"), p("residual"), p("selected"), p("weights"), p("gate"), p("up"), p("down"), p("scratch"), p("out"), M, K + 1, H, I, lib.FMT_Q4K, E + 1)
    s["lib"] = l
    torch.cuda.current_stream().synchronize()
    return s


def _run_moe(s):
    l, st = s["lib"], _stream()
    lib.check(l.sb_moe_route(st, ctypes.byref(s["route"])))
    lib.check(l.sb_moe_experts(st, ctypes.byref(s["experts"])))
    return {"out": s["out"], "selected": s["selected"], "weights": s["weights"]}


def _exact_moe(case, seed):
    s = _moe_inputs(case, seed, _device())
    M, E, K, H, I = case["rows"], case["experts"], case["top_k"], case["hidden"], case["inter"]
    x = s["x"].double()
    top, ids = torch.sort(s["scores"].double(), dim=-1, descending=True, stable=True)
    weights = torch.cat([torch.softmax(top[:, :K], -1), torch.sigmoid(x @ s["shared_gate"].double()).unsqueeze(-1)], -1)
    ids = torch.cat([ids[:, :K], torch.full((M, 1), E, device=ids.device)], -1)
    out = s["residual"].double()
    for e in torch.unique(ids).tolist():
        row, slot = (ids == e).nonzero(as_tuple=True)
        w = lambda k, n, kk: _dequant64("q4k", s[k].reshape(E + 1, n, -1)[e], kk)
        gate, up = x[row] @ w("gate", I, H).T, x[row] @ w("up", I, H).T
        y = (up * gate * torch.sigmoid(gate)) @ w("down", H, I).T
        out.index_add_(0, row, y * weights[row, slot].unsqueeze(-1))
    return {"out": out, "selected": None, "weights": weights}


def _work_moe(case):
    M, E, K, H, I = case["rows"], case["experts"], case["top_k"], case["hidden"], case["inter"]
    hit = E * (1.0 - (1.0 - K / E) ** M) + 1  # the experts that some row is expected to name, and the shared one
    return {"bytes": int(hit * 3 * I * H * 144 / 256 + M * (6 * H + 4 * E + 16 * (K + 1))), "flops": int(6 * M * (K + 1) * I * H)}


# ---- selection: the rows' next tokens and the lane's accepted drafts, from logits ----

def _prepare_select(case, seed):
    d = _device()
    l = lib.ops()
    g = _generator(seed, d)
    L, R, V = case["lanes"], case["rows"], case["vocab"]
    s = {}
    # Logits as a language model's head gives them: most tokens around zero, a few far above.
    x = torch.randn((L * ROW_SLOTS, V), generator=g, device=d) * 1.8
    heavy = torch.randint(0, V, (L * ROW_SLOTS, 64), generator=g, device=d)
    s["logits"] = x.scatter(1, heavy, 6.0 + 3.0 * torch.randn(heavy.shape, generator=g, device=d)).contiguous()
    top = s["logits"].argmax(-1).reshape(L, ROW_SLOTS)
    other = torch.randint(0, V, (L, ROW_SLOTS), generator=g, device=d)
    # A draft the target would mostly take: row r + 1 proposes what row r likes best, two times in three.
    likes = torch.cat([other[:, :1], top[:, :-1]], -1)
    s["tokens"] = torch.where(torch.rand((L, ROW_SLOTS), generator=g, device=d) < 0.67, likes, other).to(torch.int32).contiguous()
    s["uniforms"] = torch.rand((L, 80), generator=g, device=d)
    s["tree"] = _tree_tensor(L, R, seed, False, d)
    s["selected"] = torch.zeros((L, ROW_SLOTS), dtype=torch.int32, device=d)
    s["results"] = torch.zeros((L, 4), dtype=torch.int32, device=d)
    s["tickets"] = torch.zeros((L,), dtype=torch.int32, device=d)
    s["workspace"] = torch.empty(int(l.sb_sample_workspace_bytes(ROW_SLOTS * L, V)), dtype=torch.uint8, device=d)
    p = lambda k: s[k].data_ptr()
    a = lib.SbSelectAcceptArgs()
    q = a.sample
    q.logits, q.input_tokens, q.uniforms, q.selected, q.workspace = p("logits"), p("tokens"), p("uniforms"), p("selected"), p("workspace")
    q.rows, q.vocab, q.logit_stride, q.temperature, q.min_p, q.top_k, q.top_p = R, V, V, case["temperature"], case["min_p"], case["top_k"], case["top_p"]
    q.lanes = L if L > 1 else 0
    b = a.accept
    b.input_tokens, b.tree, b.tokens, b.results, b.rows, b.remaining, b.lanes = p("tokens"), p("tree"), p("selected"), p("results"), R, 0xFFFFFFFF, q.lanes
    a.tickets = p("tickets")
    s["args"], s["case"], s["lib"] = a, case, l
    torch.cuda.current_stream().synchronize()
    return s


def _run_select(s):
    lib.check(s["lib"].sb_select_accept(_stream(), ctypes.byref(s["args"])))
    return {"selected": s["selected"][:, :s["case"]["rows"]], "results": s["results"]}


def _work_select(case):
    return {"bytes": int(case["lanes"] * case["rows"] * case["vocab"] * 4), "flops": int(case["lanes"] * case["rows"] * case["vocab"] * 4)}


# ---- a whole verify step of a target from host tokens ----

def _step_config(case):
    base = target.QWEN27B if case["model"] == "27b" else target.TINY
    cfg = dict(base, layers=case["layers"], max_context=case["context"] + 1024)
    if case["lanes"] > 1:
        cfg["lanes"] = case["lanes"]
    return cfg


def _prepare_step(case, seed):
    d = _device()
    cfg = _step_config(case)
    L, R = case["lanes"], case["rows"]
    t = target.Target(**cfg)
    t.randomize(int(seed) + 1, case["context"])
    g = _generator(seed, d)
    # The last of the prompt enters as a block; then the lane is held at its position and folds six of that block's rows in
    # every pass, so that every pass does a committing step's work.
    prompt = torch.randint(0, cfg["vocab"], (L, ROW_SLOTS), generator=g, device=d).cpu().numpy().astype(np.uint32)
    if L > 1:
        t.verify_lanes(prompt, flags=target.ADVANCE | target.PROMPT)
    else:
        t.verify(prompt[0], flags=target.ADVANCE | target.PROMPT)
    t.upload(-1, "pending_rows", np.full(L, 6, np.uint32))
    tokens = torch.randint(0, cfg["vocab"], (L, R), generator=g, device=d).cpu().numpy().astype(np.uint32)
    uniforms = torch.rand((L, 80), generator=g, device=d).cpu().numpy() if case["temperature"] > 0 else None
    ptr, _ = t.tensor(-1, "logits")
    logits = torch.as_tensor(_DeviceArray(t, ptr, (L, ROW_SLOTS, cfg["vocab"]), "<f4"), device=d)
    torch.cuda.synchronize()
    return dict(case=case, target=t, tokens=tokens, uniforms=uniforms, logits=logits)


def _run_step(s):
    case, t = s["case"], s["target"]
    flags = target.GRAPH | target.KEEP_PENDING
    if case["lanes"] > 1:
        per_lane = t.verify_lanes(s["tokens"], uniforms=s["uniforms"], temperature=case["temperature"], flags=flags, stream=_stream() or None)
    else:
        per_lane = [t.verify(s["tokens"][0], uniforms=None if s["uniforms"] is None else s["uniforms"][0], temperature=case["temperature"], flags=flags, stream=_stream() or None)]
    return {"logits": s["logits"][:, :case["rows"]], "retained": [int(r[1]) for r in per_lane]}


def _work_step(case):
    c = _step_config(case)
    L, R, H, I, V, D, N = case["lanes"], case["rows"], c["hidden"], c["intermediate"], c["vocab"], c["head_dim"], case["layers"]
    attn = N // c["attention_interval"]
    gdn = N - attn
    per = {lib.FMT_Q4K: 144 / 256, lib.FMT_Q6K: 210 / 256}
    KW, VW = c["gdn_key_heads"] * GDN_DIM, c["gdn_value_heads"] * GDN_DIM
    attn_w = H * (c["q_heads"] * 2 * D + 2 * c["kv_heads"] * D) + c["q_heads"] * D * H
    gdn_w = H * (2 * KW + 2 * VW) + VW * H
    proj, down, head = attn * attn_w + gdn * gdn_w + N * 2 * H * I, N * H * I, H * V
    weights = proj * per[c["fmt_proj"]] + down * per[c["fmt_down"]] + head * per[c["fmt_head"]] + gdn * 2 * c["gdn_value_heads"] * H * 4
    kv = L * attn * case["context"] * 2 * c["kv_heads"] * (D + 2)
    state = L * gdn * 8 * c["gdn_value_heads"] * GDN_DIM * GDN_DIM
    flops = 2 * L * R * (proj + down + head) + 4 * L * R * attn * case["context"] * c["q_heads"] * D
    return {"bytes": int(weights + kv + state + L * R * V * 4), "flops": int(flops)}


# ---- the cases' calls ----

_PREPARE = dict(ffn=_prepare_ffn, attention=_prepare_attention, gdn=_prepare_gdn, moe=_prepare_moe, select=_prepare_select, step=_prepare_step)
_RUN = dict(ffn=_run_ffn, attention=_run_attention, gdn=_run_gdn, moe=_run_moe, select=_run_select, step=_run_step)
_WORK = dict(ffn=_work_ffn, attention=_work_attention, gdn=_work_gdn, moe=_work_moe, select=_work_select, step=_work_step)
_EXACT = dict(ffn=_exact_ffn, attention=_exact_attention, gdn=_exact_gdn, moe=_exact_moe)


def prepare(case, seed):
    return dict(kind=case["kind"], state=_PREPARE[case["kind"]](case, seed))


def run(state):
    return _RUN[state["kind"]](state["state"])


def work(case):
    return _WORK[case["kind"]](case)


def exact(case, seed):
    """None for selected tokens (whole numbers, which stay what they are) and for whole steps: their weights are the library's
    own seeded synthetic ones, which plain torch does not make; the step's layers have their 64-bit values in the other cases."""
    return _EXACT[case["kind"]](case, seed) if case["kind"] in _EXACT else None


def tolerance(case):
    if case["kind"] == "select":
        return "exact"
    if case["kind"] == "step":
        # Activations are bf16 between layers and keys and values are stored as eight-bit codes: one changed rounding in an
        # early layer reaches the logits through all that follow (the 27B shape with its attention sums in another order in
        # one layer of four: 7.5e-4, 5e-3 at most).
        return {"rel": 4e-3, "max": 0.03, "differ": 0.0}
    # bf16 results of fp32 sums over halves (an attention layer with its sums in another order: 8.7e-4, 0.07 at most).
    return {"rel": 4e-3, "max": 0.28, "differ": 0.0}
