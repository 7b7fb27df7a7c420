"""Workloads that stand for how this library is used, for timing a change against another version.

A case is a dict of plain values.  prepare(case, seed) makes what a program holds before the call (weights in an
expert arena, routers, token rows, plans, a captured graph), run(state) makes one pass through the public entry
points of libq4cuda.so, work(case) says what a pass cannot do without and tolerance(case) how far two correct
implementations may be apart.

Shapes are those of the benchmark and the tests: hidden 2048, expert width 512, 512 experts, top-10 plus one shared
expert, and the other widths the tests use.  A model has 48 such layers; a pass here walks up to 12 of them, enough
weights (0.7 GB a layer) that no layer's are in the L2 cache when its turn comes.  Every layer of a pass has token
rows of its own, as it has in a model where attention sits between two MoE layers; only the stack call chains its
layers, which is what that call does.
"""
import ctypes as C
import gc

import numpy as np
import torch

import __graft_entry__ as entry

EPS = 1e-6
F32, Q4_K, Q5_K, Q6_K, IQ3_XXS, IQ4_NL, IQ3_S, IQ2_S, IQ4_XS, Q2_0 = 0, 12, 13, 14, 18, 20, 21, 22, 23, 42
# type id: (bytes per block, values per block, offset of the fp16 scale, offset of the fp16 minimum)
BLOCKS = {Q4_K: (144, 256, 0, 2), Q5_K: (176, 256, 0, 2), Q6_K: (210, 256, 208, None), IQ3_XXS: (98, 256, 0, None),
          IQ4_NL: (18, 32, 0, None), IQ3_S: (110, 256, 0, None), IQ2_S: (82, 256, 0, None),
          IQ4_XS: (136, 256, 0, None), Q2_0: (18, 64, 0, None)}
# gate+up and down formats of the mixed expert packs that deployed models use
MIXES = [(IQ2_S, IQ4_NL), (IQ3_XXS, Q2_0), (IQ3_S, IQ4_NL), (IQ4_XS, IQ4_XS), (IQ2_S, Q2_0), (IQ4_NL, IQ4_NL), (IQ3_S, IQ3_S)]
BATCH_MIXES = [(IQ4_XS, IQ4_NL), (IQ4_NL, IQ4_NL), (IQ3_S, IQ4_NL), (IQ4_XS, IQ4_XS)]


def row_bytes(ty, cols):
    bs, vals = BLOCKS[ty][:2]
    return cols // vals * bs


def listed():
    model = {"experts": 512, "topk": 10, "embd": 2048, "ff": 512}
    return [
        # one token through consecutive layers in one call, the decode loop of the benchmark
        dict(model, name="decode stack", kind="stack", tokens=1, layers=12),
        # one token, one call a layer on device rows: a model with attention between the layers
        dict(model, name="decode by layer", kind="layers", tokens=1, layers=12),
        # the same for a caller whose rows are on the host: row in, row out, every layer
        dict(model, name="decode host rows", kind="host", tokens=1, layers=12),
        # the engine's own sequence of small calls for one token on experts of mixed formats, as a graph
        dict(model, name="decode mixed formats", kind="exec", tokens=1, layers=12, gu=IQ2_S, down=IQ4_NL),
        # speculative decoding: four tokens are verified together
        dict(model, name="verify 4 tokens", kind="batch", tokens=4, layers=12),
        # the engine's verify window over slot lists that it routed itself
        dict(model, name="verify window lists", kind="window", tokens=3, layers=12),
        # batched decode, the benchmark's 64 tokens
        dict(model, name="batch 64", kind="batch", tokens=64, layers=12),
        # a small batch on experts in the 4-bit formats
        dict(model, name="batch 33 4-bit", kind="batch4", tokens=33, layers=6, gu=IQ4_XS, down=IQ4_NL),
        # prefill: a ragged last chunk, the benchmark's chunk with skewed expert popularity, a long prompt
        dict(model, name="prefill 777", kind="prefill", tokens=777, layers=1, skew=0.0),
        dict(model, name="prefill 2048 skewed", kind="prefill", tokens=2048, layers=1, skew=1.1),
        dict(model, name="prefill 8192", kind="prefill", tokens=8192, layers=1, skew=0.0),
        # dense projections of a verify window (attention and shared matrices) in a K-quant format
        {"name": "dense 4 rows", "kind": "dense", "tokens": 4, "layers": 16, "rows": 4096, "embd": 2048, "gu": Q4_K},
    ]


def log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["stack", "layers", "host", "exec", "window", "batch", "batch", "batch", "batch4", "prefill", "prefill",
                       "prefill", "dense"])
    if kind == "dense":
        return {"kind": kind, "tokens": rng.randint(2, 8), "layers": rng.randint(4, 16), "rows": 256 * rng.randint(2, 20),
                "embd": rng.choice([1024, 2048, 2560, 4096]), "gu": rng.choice([Q4_K, Q5_K, Q6_K, IQ4_XS, IQ4_NL])}
    experts = log_int(rng, 48, 512)
    case = {"experts": experts, "topk": rng.randint(4, 10), "embd": 2048, "ff": 512, "kind": kind, "tokens": 1,
            "layers": rng.randint(3, 12)}
    if kind == "stack":
        return case
    if rng.random() < 0.35:   # the other widths
        case["embd"], case["ff"] = rng.choice([(1024, 256), (2048, 768), (2560, 512), (1024, 512), (2048, 1024)])
    if kind in ("exec", "batch4"):
        case["gu"], case["down"] = rng.choice(MIXES if kind == "exec" else BATCH_MIXES)
    if kind == "window":
        case["tokens"] = rng.randint(2, 8)
    if kind == "batch":
        case["tokens"] = log_int(rng, 2, 256)
        case["layers"] = rng.randint(2, 12 if case["tokens"] <= 64 else 4)
    if kind == "batch4":
        case["tokens"] = log_int(rng, 2, 128)
        case["layers"] = rng.randint(2, 4)
    if kind == "prefill":
        wide = case["embd"] * case["ff"] > 2048 * 512
        case["tokens"], case["layers"] = log_int(rng, 257, 4096 if wide else 8000), 1
        case["skew"] = rng.choice([0.0, 0.0, 1.1])
    return case


def arrays(case):
    """Bytes of one expert's gate and up rows and of its down rows."""
    gu, dn = case.get("gu", IQ3_S), case.get("down", IQ3_S)
    return 2 * case["ff"] * row_bytes(gu, case["embd"]), case["embd"] * row_bytes(dn, case["ff"])


def distinct(case):
    """Expected number of experts that a layer's tokens pick, from sampled router logits."""
    rng = np.random.default_rng(1)
    logits = rng.standard_normal((512, case["experts"])) * 0.9 + zipf_bias(case["experts"], case.get("skew", 0.0))
    picked = np.argsort(-logits, axis=1)[:, :case["topk"]]
    share = np.bincount(picked.ravel(), minlength=case["experts"]) / 512.0
    return float((1 - (1 - share) ** case["tokens"]).sum())


def work(case):
    t, layers, embd = case["tokens"], case["layers"], case["embd"]
    if case["kind"] == "dense":
        n = case["rows"]
        return {"bytes": layers * (n * row_bytes(case["gu"], embd) + 4 * t * (n + embd)), "flops": 2.0 * layers * t * n * embd}
    shared = 0 if case["kind"] == "exec" else 1
    routed = case["kind"] != "window"
    weights = (distinct(case) + shared) * sum(arrays(case))
    router = 4 * case["experts"] * embd if routed else 0
    flops = 2.0 * t * (3 * embd * case["ff"] * (case["topk"] + shared) + (case["experts"] * embd if routed else 0))
    return {"bytes": layers * (weights + router + 8 * t * embd), "flops": layers * flops}


def tolerance(case):
    if case["kind"] == "stack":
        return "exact"    # a layer's row is the next one's input: the order of every sum is part of this call's result
    if case["kind"] == "dense":
        return {"rel": 1e-5}
    # Hidden values are quantised to 8 bits between the two products: a value that differs in its last bit may round
    # to the neighbouring step, and such a step moves a row by up to 1e-3 (the bound of the tests).  Picks: near-ties.
    return {"rel": 1e-3, "differ": 0.01}


# ------------------------------------------------------------------ what a program has in hand

_lib = None


def library():
    global _lib
    if _lib is None:
        pkg = entry.load_package()
        _lib = pkg.capi.load()
        if not _lib.q4_hip_init():
            raise RuntimeError("q4_hip_init failed")
    return _lib


def must(ok, what):
    if not ok:
        raise RuntimeError(what + " refused")


class StackLayer(C.Structure):
    _fields_ = [("base", C.c_void_p), ("norm", C.c_void_p), ("router", C.c_void_p)]


class State:
    """Buffers, plans and graph of one prepared case; gives back what the library holds for it."""

    def __init__(self, case):
        self.case, self.lib = case, library()
        self.arena, self.plans, self.stack, self.graph, self.host = None, [], None, None, []

    def __del__(self):
        lib = self.lib
        lib.q4_hip_sync()
        if self.graph:
            lib.q4_hip_graph_free(self.graph)
        for p in self.plans:
            lib.q4_cuda_decode_plan_free(p)
        if self.stack:
            lib.q4_cuda_decode_stack_free(self.stack)
        for p in self.host:
            lib.q4_hip_host_free_coh(p)
        if self.arena is not None:
            lib.q4_hip_experts_free_a(self.arena)


def zipf_bias(n, s):
    p = np.arange(1, n + 1, dtype=np.float64) ** -s
    return np.log(p / p.sum()) if s else np.zeros(n)


def random_blocks(gen, ty, nbytes):
    """Blocks of a format with every payload byte uniform and fp16 scales of the magnitudes that the tests use."""
    bs, _, od, om = BLOCKS[ty]
    b = torch.randint(0, 256, (nbytes // bs, bs), dtype=torch.uint8, device="cuda", generator=gen)
    small = ty in (Q4_K, Q5_K, Q6_K)
    d = torch.randn(len(b), device="cuda", generator=gen).abs() * 2.0 ** (-8 if small else -6)
    b[:, od:od + 2] = d.half().view(torch.uint8).view(-1, 2)
    if om is not None:
        m = torch.randn(len(b), device="cuda", generator=gen).abs() * 2.0 ** -9
        b[:, om:om + 2] = m.half().view(torch.uint8).view(-1, 2)
    return b


def fill_arena(s, gen, seed):
    """An arena of layers x (experts + shared) packs."""
    case, lib = s.case, s.lib
    gu, dn = case.get("gu", IQ3_S), case.get("down", IQ3_S)
    gu_bytes, dn_bytes = arrays(case)
    s.pack, s.slots = gu_bytes + dn_bytes, case["experts"] + 1
    s.og, s.ou, s.od = 0, gu_bytes // 2, gu_bytes
    n = case["layers"] * s.slots
    plain = gu == IQ3_S and dn == IQ3_S
    free = [a for a in range(4) if not lib.q4_hip_experts_base_a(a)]
    if not free:
        gc.collect()
        free = [a for a in range(4) if not lib.q4_hip_experts_base_a(a)]
    lib.q4_cuda_set_tiled_default(1 if plain else 0)
    ok = bool(free) and lib.q4_hip_experts_alloc_a(free[0], n, s.pack)
    lib.q4_cuda_set_tiled_default(1)
    if not ok:
        raise MemoryError("out of memory: an arena of %d slots" % n)
    s.arena = free[0]
    s.base, s.stride = lib.q4_hip_experts_base_a(s.arena), lib.q4_hip_experts_stride_a(s.arena)
    if plain:
        must(lib.q4_cuda_synth_iq3s(s.base, n * (s.pack // 110), seed), "synth")
        must(lib.q4_cuda_experts_retile_a(s.arena, 0, n), "retile")
        return
    for l in range(case["layers"]):
        packs = torch.empty(s.slots, s.pack, dtype=torch.uint8, device="cuda")
        packs[:, :gu_bytes] = random_blocks(gen, gu, s.slots * gu_bytes).view(s.slots, -1)
        packs[:, gu_bytes:] = random_blocks(gen, dn, s.slots * dn_bytes).view(s.slots, -1)
        torch.cuda.synchronize()
        must(lib.q4_hip_copy_async(s.base + l * s.slots * s.stride, packs.data_ptr(), packs.numel() // 4), "copy")
        lib.q4_hip_sync()


def capture(s, enqueue):
    """The pass as a CUDA graph, which is how a decode loop replays it."""
    lib = s.lib
    must(lib.q4_hip_graph_begin() == 1, "graph capture")
    try:
        enqueue()
    finally:
        s.graph = lib.q4_hip_graph_end()
    must(s.graph, "graph")


def prepare(case, seed):
    s = State(case)
    lib, kind, t, layers, embd = s.lib, case["kind"], case["tokens"], case["layers"], case["embd"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)

    def randn(*shape):
        return torch.randn(*shape, device="cuda", generator=gen)

    if kind == "dense":
        n = case["rows"]
        s.w = random_blocks(gen, case["gu"], layers * n * row_bytes(case["gu"], embd))
        s.x, s.y = randn(layers, t, embd), torch.empty(layers, t, n, device="cuda")
        step = n * row_bytes(case["gu"], embd)

        def dense():
            for l in range(layers):
                must(lib.q4_mmvq_n(case["gu"], s.w.data_ptr() + l * step, n, embd, s.x[l].data_ptr(), s.y[l].data_ptr(), 1.0, t),
                     "q4_mmvq_n")
        torch.cuda.synchronize()
        capture(s, dense)
        s.out = {"y": s.y}
        return s

    e, k, ff = case["experts"], case["topk"], case["ff"]
    fill_arena(s, gen, seed)
    s.router = randn(layers, e, embd) * 0.02
    s.norm = 1.0 + 0.1 * randn(layers, embd)
    s.x = randn(layers, t, embd)
    if case.get("skew"):   # coordinate 0 is the same in every token and carries the experts' popularity
        s.x[..., 0] = 4.0
        s.norm[:, 0] = 1.0
        bias = zipf_bias(e, case["skew"]) / (4.0 / np.sqrt((16.0 + embd - 1) / embd))
        s.router[..., 0] = torch.tensor(bias, dtype=torch.float32, device="cuda")
    s.y = torch.empty(layers, t, embd, device="cuda")
    s.ids = torch.empty(layers, t, k, dtype=torch.int32, device="cuda")
    s.wts = torch.empty(layers, t, k, device="cuda")
    s.out = {"y": s.y, "ids": s.ids, "wts": s.wts}
    at = [s.base + l * s.slots * s.stride for l in range(layers)]
    torch.cuda.synchronize()

    if kind == "stack":
        arr = (StackLayer * layers)()
        for l in range(layers):
            arr[l].base, arr[l].norm, arr[l].router = at[l], s.norm[l].data_ptr(), s.router[l].data_ptr()
        s.stack = lib.q4_cuda_decode_stack_plan(arr, layers, s.stride, s.og, s.ou, s.od, e, EPS, e, k, embd, ff)
        must(s.stack, "q4_cuda_decode_stack_plan")
        s.out = {"y": s.y[0], "ids": s.ids, "wts": s.wts}
        s.args = (s.stack, s.x.data_ptr(), s.y.data_ptr(), s.ids.data_ptr(), s.wts.data_ptr())
    elif kind in ("layers", "host"):
        for l in range(layers):
            s.plans.append(lib.q4_cuda_decode_plan(at[l], s.stride, s.og, s.ou, s.od, e, s.norm[l].data_ptr(), EPS,
                                                   s.router[l].data_ptr(), e, k, embd, ff))
            must(s.plans[-1], "q4_cuda_decode_plan")
        if kind == "layers":
            s.args = [(s.plans[l], s.x[l].data_ptr(), s.y[l].data_ptr(), s.ids[l].data_ptr(), s.wts[l].data_ptr())
                      for l in range(layers)]
        else:
            s.hx = s.x.view(layers, embd).cpu().numpy()
            p = lib.q4_hip_host_alloc_coh(layers * embd * 4)
            must(p, "q4_hip_host_alloc_coh")
            s.host.append(p)
            s.hy = np.ctypeslib.as_array((C.c_float * (layers * embd)).from_address(p)).reshape(layers, embd)
            s.args = [(s.plans[l], s.hx[l].ctypes.data, p + l * embd * 4) for l in range(layers)]
    elif kind == "exec":
        s.xn, s.logits = torch.empty(layers, embd, device="cuda"), torch.empty(layers, e, device="cuda")
        s.h = torch.empty(64 * ff, device="cuda")
        s.n = torch.tensor([k], dtype=torch.int32, device="cuda")
        gu, dn = case["gu"], case["down"]

        def sequence():
            for l in range(layers):
                xn, lg, y = s.xn[l].data_ptr(), s.logits[l].data_ptr(), s.y[l].data_ptr()
                ids, wts = s.ids[l].data_ptr(), s.wts[l].data_ptr()
                must(lib.q4_hip_grouped_rms(s.x[l].data_ptr(), s.norm[l].data_ptr(), xn, embd, 1, EPS), "q4_hip_grouped_rms")
                must(lib.q4_hip_gemv_dd(F32, s.router[l].data_ptr(), e, embd, xn, lg, 1.0), "q4_hip_gemv_dd")
                must(lib.q4_hip_fill(y, 0.0, embd), "q4_hip_fill")
                must(lib.q4_hip_softmax_topk_launch(lg, e, k, ids, wts), "q4_hip_softmax_topk_launch")
                must(lib.q4_hip_moe_exec_dev(at[l], s.stride, ids, wts, s.n.data_ptr(), gu, s.og, gu, s.ou, dn, s.od, xn,
                                             s.h.data_ptr(), None, None, y, ff, embd, embd), "q4_hip_moe_exec_dev")
        torch.cuda.synchronize()
        capture(s, sequence)
    elif kind == "window":
        # the token's picks (distinct), then the shared expert with weight 1, in lists of 64
        pick = torch.rand(layers, t, e, device="cuda", generator=gen).topk(k, dim=2).indices
        s.es = torch.full((layers, t, 64), -1, dtype=torch.int32, device="cuda")
        s.ew = torch.zeros(layers, t, 64, device="cuda")
        s.es[..., :k], s.es[..., k] = pick.int(), e
        s.ew[..., :k] = torch.softmax(randn(layers, t, k), 2)
        s.ew[..., k] = 1.0
        s.nh = torch.full((t,), k + 1, dtype=torch.int32, device="cuda")
        s.h = torch.empty(t * 64 * ff, device="cuda")

        def window():
            for l in range(layers):
                must(lib.q4_hip_fill(s.y[l].data_ptr(), 0.0, t * embd), "q4_hip_fill")
                must(lib.q4_hip_moe_exec_win(at[l], s.stride, s.es[l].data_ptr(), s.ew[l].data_ptr(), s.nh.data_ptr(), t, IQ3_S,
                                             s.og, IQ3_S, s.ou, IQ3_S, s.od, s.x[l].data_ptr(), s.h.data_ptr(),
                                             s.y[l].data_ptr(), ff, embd, embd), "q4_hip_moe_exec_win")
        torch.cuda.synchronize()
        capture(s, window)
        s.out = {"y": s.y}
    else:
        nb = lib.q4_cuda_moe_layer_n_ws_bytes(t, k, e, embd, ff)
        s.ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
        tail = [(s.x[l].data_ptr(), s.norm[l].data_ptr(), EPS, s.router[l].data_ptr(), e, k, embd, ff, t, s.y[l].data_ptr(),
                 s.ids[l].data_ptr(), s.wts[l].data_ptr(), s.ws.data_ptr(), nb) for l in range(layers)]

        if kind == "batch4":
            def enqueue():
                for l in range(layers):
                    must(lib.q4_cuda_moe_layer_nt(at[l], s.stride, case["gu"], s.og, s.ou, case["down"], s.od, e, *tail[l]),
                         "q4_cuda_moe_layer_nt")
        else:
            def enqueue():
                for l in range(layers):
                    must(lib.q4_cuda_moe_layer_n(at[l], s.stride, s.og, s.ou, s.od, e, *tail[l]), "q4_cuda_moe_layer_n")
        torch.cuda.synchronize()
        if kind == "prefill":
            s.enqueue = enqueue   # a prompt's chunk is a plain call: its length is another one each time
        else:
            capture(s, enqueue)
    lib.q4_hip_sync()
    return s


def run(s):
    lib, kind = s.lib, s.case["kind"]
    if s.graph:
        must(lib.q4_hip_graph_launch(s.graph), "q4_hip_graph_launch")
    elif kind == "stack":
        must(lib.q4_cuda_decode_stack_dev(*s.args), "q4_cuda_decode_stack_dev")
    elif kind == "layers":
        for a in s.args:
            must(lib.q4_cuda_decode_plan_dev(*a), "q4_cuda_decode_plan_dev")
    elif kind == "host":
        for a in s.args:
            must(lib.q4_cuda_decode_plan_host(*a), "q4_cuda_decode_plan_host")
        return {"y": s.hy}
    else:
        s.enqueue()
    return s.out
