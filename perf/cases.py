"""The library's work as its users have it done, for timing: what `bench.py` runs, its
neighbours in size, and the steps that a serving loop puts together from the same entry
points.  A case names a kind of step and its sizes; `prepare` makes what a host program
holds before the step, `run` takes the step once.

    decode   one token through every layer of one sequence: append and attention over an
             fp16 or an e4m3 cache.  The cursor lives on the device and the host replays one
             captured graph per token, as the engine does (crates/whetstone-kernels/cuda/graph.cu)
    chunk    several tokens of one sequence, layer by layer, launched as they come (the
             chunk's start is a host value): drafts under verification, chunked prompts
    batch    chunked prompts of several sequences of one length in one launch per step
    paged    a ragged step over the paged cache: drafts of many sequences, or prompts
             that fill beside sequences that decode
    proj     the projections either side of the attention, weights of several layers in turn
    block    projection, append, attention and output projection of a chunk step
"""

from __future__ import annotations

import math

import torch

from whetstone_b200 import chunk, decode, paged, workloads

SHAPES = {s.name: s for s in (workloads.QWEN25_05B, workloads.QWEN25_7B, workloads.QWEN3_8B)}
HIDDEN = {"qwen2.5-0.5b": 896, "qwen2.5-7b": 3584, "qwen3-8b": 4096}
EPS = 1e-6
E4M3_SCALE = 0.0625     # a stored byte times this is the value: keys and values up to 28


def listed():
    return [
        # The smallest step: one token of the small model behind a short prompt.  Every
        # launch is a few microseconds, so their number and latency are the cost.
        {"name": "decode-05b-512", "kind": "decode", "shape": "qwen2.5-0.5b", "layers": 24,
         "rows": 513, "max_seq": 1024, "cache": "fp16"},
        # One token behind a long context, cache full: the benchmark's headline.
        {"name": "decode-7b-32k", "kind": "decode", "shape": "qwen2.5-7b", "layers": 28,
         "rows": 32768, "max_seq": 32768, "cache": "fp16"},
        # The same from the 8-bit cache, somewhere inside its capacity.
        {"name": "decode-7b-e4m3-20k", "kind": "decode", "shape": "qwen2.5-7b", "layers": 28,
         "rows": 20011, "max_seq": 32768, "cache": "e4m3"},
        # One sequence's draft tokens verified in one go: a handful of rows, all layers.
        {"name": "chunk-7b-drafts", "kind": "chunk", "shape": "qwen2.5-7b", "layers": 28,
         "start": 4099, "n": 5, "steps": 1, "max_seq": 8192},
        # A prompt read in chunks, small model: eight short steps that depend on each other.
        {"name": "chunk-05b-prompt", "kind": "chunk", "shape": "qwen2.5-0.5b", "layers": 4,
         "start": 0, "n": 256, "steps": 8, "max_seq": 2048},
        # Four long prompts read together, head norm, one layer of all sixteen steps.
        {"name": "batch-8b-4x8192", "kind": "batch", "shape": "qwen3-8b", "n_seq": 4,
         "start": 0, "n": 512, "steps": 16, "max_seq": 8192},
        # Speculative verification of a batch: five rows each of sixteen ragged sequences.
        {"name": "paged-7b-verify", "kind": "paged", "shape": "qwen2.5-7b", "layers": 4,
         "n_seq": 16, "len_lo": 1024, "len_hi": 16384, "drafts": 5, "fills": 0, "fill": 0},
        # A serving step: two sequences read 300 prompt rows each beside six that verify.
        {"name": "paged-7b-mixed", "kind": "paged", "shape": "qwen2.5-7b", "layers": 4,
         "n_seq": 8, "len_lo": 512, "len_hi": 8192, "drafts": 4, "fills": 2, "fill": 300},
        # The batch's projections of a verification step: 16 x 5 rows.
        {"name": "proj-7b-fp16-80", "kind": "proj", "shape": "qwen2.5-7b", "weights": "fp16",
         "layers": 8, "n": 80},
        # One sequence's drafts through the packed weights the engine ships.
        {"name": "proj-7b-int4-5", "kind": "proj", "shape": "qwen2.5-7b", "weights": "int4",
         "layers": 28, "n": 5},
        # The whole attention block in the middle of the long prompts, either weight format.
        {"name": "block-8b-fp16", "kind": "block", "shape": "qwen3-8b", "weights": "fp16",
         "layers": 4, "n_seq": 4, "start": 4096, "n": 512, "max_seq": 8192},
        {"name": "block-8b-int4", "kind": "block", "shape": "qwen3-8b", "weights": "int4",
         "layers": 4, "n_seq": 3, "start": 2500, "n": 509, "max_seq": 4096},
    ]


# ------------------------------------------------------------------------- more cases

def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def _capacity(rng, rows):
    """A cache is allocated before it fills: up to four times the rows, in steps of 256."""
    return -(-int(rows * rng.uniform(1.0, 4.0)) // 256) * 256


def _draw_one(rng):
    kind = rng.choice(["decode", "decode", "chunk", "batch", "paged", "proj", "proj", "block"])
    shape = rng.choice(sorted(SHAPES))
    if kind == "decode":
        cache = rng.choice(["fp16", "e4m3"]) if SHAPES[shape].head_dim == 128 else "fp16"
        rows = _log(rng, 64, 65536)
        return {"kind": kind, "shape": shape, "layers": rng.randint(4, 28), "rows": rows,
                "max_seq": _capacity(rng, rows), "cache": cache}
    if kind == "chunk":
        n = _log(rng, 2, 1024)
        start, steps = rng.choice([0, _log(rng, 16, 16384)]), rng.randint(1, 6)
        return {"kind": kind, "shape": shape, "layers": rng.randint(1, 12), "start": start, "n": n,
                "steps": steps, "max_seq": _capacity(rng, start + n * steps)}
    if kind == "batch":
        n, n_seq, steps = _log(rng, 64, 1024), rng.randint(2, 8), rng.randint(1, 6)
        start = rng.choice([0, _log(rng, 16, 8192)])
        return {"kind": kind, "shape": shape, "n_seq": n_seq, "start": start, "n": n,
                "steps": steps, "max_seq": _capacity(rng, start + n * steps)}
    if kind == "paged":
        n_seq = rng.randint(2, 24)
        lo = _log(rng, 64, 4096)
        fills = rng.choice([0, 0, rng.randint(1, min(3, n_seq))])
        return {"kind": kind, "shape": shape, "layers": rng.randint(1, 4), "n_seq": n_seq,
                "len_lo": lo, "len_hi": lo * rng.randint(1, 8), "drafts": rng.randint(1, 8),
                "fills": fills, "fill": _log(rng, 16, 512) if fills else 0}
    if kind == "proj":
        return {"kind": kind, "shape": shape, "weights": rng.choice(["fp16", "int4"]),
                "layers": rng.randint(4, 28), "n": _log(rng, 2, 2048)}
    n, n_seq = _log(rng, 128, 1024), rng.randint(1, 6)
    start = rng.choice([0, _log(rng, 16, 4096)])
    return {"kind": kind, "shape": shape, "weights": rng.choice(["fp16", "int4"]),
            "layers": rng.randint(1, 6), "n_seq": n_seq, "start": start, "n": n,
            "max_seq": _capacity(rng, start + n)}


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 6e12, w["flops"] / 1e15)


def _state_bytes(case):
    """The caches, and the scratch that the paged entry point asks for."""
    s = SHAPES[case["shape"]]
    if case["kind"] == "paged":
        n = max(case["drafts"], case["fill"])
        return 4 * paged.verify_scratch_floats(case["n_seq"], n, s.n_q, s.n_kv, s.head_dim,
                                               case["len_hi"] + n)
    return (case.get("layers", 1) * case.get("n_seq", 1) * case.get("max_seq", 0) * s.n_kv
            * s.head_dim * 4)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        case = _draw_one(rng)
        if _cost(case) <= most and _state_bytes(case) <= 8 << 30:   # several states fit the card
            return case


# ----------------------------------------------------------------------------- inputs

class _Inputs:
    """Values on the GPU, from the seed alone."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, shape, scale=1.0, dtype=torch.float16):
        x = torch.empty(shape, dtype=dtype, device="cuda").normal_(generator=self.gen)
        return x if scale == 1.0 else x.mul_(scale)

    def rows(self, shape):
        """Projection outputs: numbers that fp16 holds, in the fp32 buffer of the ABI."""
        return self.normal(shape).float()

    def e4m3(self, shape):
        """N(0, 1) under E4M3_SCALE, rounded to e4m3 (no NaN: the scaled values stay below 448)."""
        out = torch.empty(shape, dtype=torch.uint8, device="cuda")
        for layer in out:
            x = self.normal(layer.shape).div_(E4M3_SCALE).clamp_(-448, 448)
            layer.copy_(x.to(torch.float8_e4m3fn).view(torch.uint8))
        return out

    def norm(self, s):
        """Head-norm gains of the one model that has them."""
        if s.name != "qwen3-8b":
            return None
        gain = lambda: (1 + self.normal((s.head_dim,), 0.02).float()).half()  # noqa: E731
        return decode.QkNorm(gain(), gain(), EPS)

    def weights(self, kind, in_f, out_f):
        """(arrays of one projection): fp16 rows, or the packed int4 arrays with the scales
        that give weights of about the same size."""
        if kind == "fp16":
            return (self.normal((out_f, in_f), in_f ** -0.5),)
        groups = out_f * in_f // 32
        ints = lambda lo, hi, n, dt: torch.randint(lo, hi, (n,), dtype=dt, device="cuda",  # noqa: E731
                                                   generator=self.gen)
        qw = ints(-2 ** 31, 2 ** 31, groups * 4, torch.int64).to(torch.int32)
        si = (ints(1, 9, groups, torch.int32) | (ints(0, 16, groups, torch.int32) << 4)).to(torch.uint8)
        sb = torch.empty((out_f, 2), dtype=torch.float32, device="cuda")
        sb[:, 0].uniform_(0.002, 0.003, generator=self.gen)
        sb[:, 1].uniform_(0.008, 0.014, generator=self.gen)
        return qw, si, (sb * (32 / in_f ** 0.5)).half()


def prepare(case, seed):
    s = SHAPES[case["shape"]]
    return {"decode": _prepare_decode, "chunk": _prepare_chunk, "batch": _prepare_batch,
            "paged": _prepare_paged, "proj": _prepare_proj,
            "block": _prepare_block}[case["kind"]](case, s, _Inputs(seed))


def _prepare_decode(case, s, make):
    layers, e4m3 = case["layers"], case["cache"] == "e4m3"
    shape = (layers, s.n_kv, case["max_seq"], s.head_dim)
    keys, values = (make.e4m3 if e4m3 else make.normal)(shape), (make.e4m3 if e4m3 else make.normal)(shape)
    caches = []
    for i in range(layers):
        if e4m3:
            c = decode.KvCacheFp8(s.n_kv, s.n_q, s.head_dim, case["max_seq"], E4M3_SCALE, E4M3_SCALE)
        else:
            c = decode.KvCache(s.n_kv, s.n_q, s.head_dim, case["max_seq"])
        c.k, c.v = keys[i], values[i]       # the layers' caches lie end to end
        caches.append(c)
    qkv = make.rows((layers, s.qkv_width))
    out = torch.zeros((layers, s.n_q * s.head_dim), dtype=torch.float16, device="cuda")
    table = decode.RopeTable(case["max_seq"], s.head_dim, s.theta)
    cursor, norm = decode.DeviceCursor(case["rows"] - 1), make.norm(s)

    def token():
        for i, c in enumerate(caches):
            if e4m3:
                decode.rope_cache_fp8(qkv[i], c, table, s.n_q, cursor, qk_norm=norm)
                decode.attn_decode_fp8(qkv[i], c, out[i], s.n_q, cursor)
            else:
                decode.rope_cache(qkv[i], c, table, s.n_q, cursor, norm)
                decode.attn_decode(qkv[i], c, out[i], s.n_q, cursor)

    token()                                 # outside the capture first, as the ABI asks
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        token()
    return {"case": case, "step": graph.replay, "results": (out, qkv, keys, values),
            "keep": (graph, caches, table, cursor, norm)}


def _prepare_chunk(case, s, make):
    layers, n, steps = case["layers"], case["n"], case["steps"]
    shape = (layers, s.n_kv, case["max_seq"], s.head_dim)
    keys, values = make.normal(shape), make.normal(shape)
    caches = []
    for i in range(layers):
        c = decode.KvCache(s.n_kv, s.n_q, s.head_dim, case["max_seq"])
        c.k, c.v = keys[i], values[i]
        caches.append(c)
    qkv = make.rows((steps, layers, n, s.qkv_width))
    out = torch.zeros((steps, layers, n, s.n_q * s.head_dim), dtype=torch.float16, device="cuda")
    table, norm = decode.RopeTable(case["max_seq"], s.head_dim, s.theta), make.norm(s)

    def step():
        for j in range(steps):
            pos0 = case["start"] + j * n
            for i, c in enumerate(caches):
                chunk.rope_cache(qkv[j, i], c, table, s.n_q, pos0, n, norm)
                chunk.attn(qkv[j, i], c, out[j, i], s.n_q, pos0, n)

    return {"case": case, "step": step, "results": (out, qkv, keys, values)}


def _batch_cache(case, s, make):
    cache = chunk.KvCacheBatch(case["n_seq"], s.n_kv, s.head_dim, case["max_seq"])
    cache.k, cache.v = make.normal(cache.k.shape), make.normal(cache.v.shape)
    return cache


def _starts(case, step=0):
    return torch.full((case["n_seq"],), case["start"] + step * case["n"], dtype=torch.int32,
                      device="cuda")


def _prepare_batch(case, s, make):
    n_seq, n, steps = case["n_seq"], case["n"], case["steps"]
    cache = _batch_cache(case, s, make)
    qkv = make.rows((steps, n_seq, n, s.qkv_width))
    out = torch.zeros((steps, n_seq, n, s.n_q * s.head_dim), dtype=torch.float16, device="cuda")
    starts = [_starts(case, j) for j in range(steps)]
    table, norm = decode.RopeTable(case["max_seq"], s.head_dim, s.theta), make.norm(s)

    def step():
        for j in range(steps):
            chunk.rope_cache_batch(qkv[j], cache, table, s.n_q, starts[j], n, norm)
            chunk.attn_batch(qkv[j], cache, out[j], s.n_q, starts[j], n)

    return {"case": case, "step": step, "results": (out, qkv, cache.k, cache.v)}


def _paged_step(case):
    """(lengths, rows of the step) per sequence: evenly spread lengths in an order that does
    not rise, the prompts that fill taken from the whole range."""
    n_seq = case["n_seq"]
    span = case["len_hi"] - case["len_lo"]
    lengths = [case["len_lo"] + span * ((7 * i + 3) % n_seq) // max(1, n_seq - 1) for i in range(n_seq)]
    rows = [case["fill"] if i < case["fills"] else case["drafts"] for i in range(n_seq)]
    return [min(x, case["len_hi"]) for x in lengths], rows


def _prepare_paged(case, s, make):
    lengths, rows = _paged_step(case)
    max_len = max(a + b for a, b in zip(lengths, rows))
    pages = sum(-(-(a + b) // paged.PAGE_SIZE) for a, b in zip(lengths, rows))
    kv = paged.PagedKvManager(pages, max_len)
    ids = workloads.c5_fill_manager(kv, lengths)
    entries = sorted(zip(ids, rows), key=lambda e: -kv.length(e[0]))    # longest context first
    plan = kv.build_step(entries)
    caches = []
    for _ in range(case["layers"]):
        c = paged.PagedKvCache(pages, s.n_kv, s.head_dim, plan.n_seq, kv.max_pages)
        c.k.normal_(generator=make.gen)
        c.v.normal_(generator=make.gen)
        pos0, cu = plan.upload(c)
        caches.append(c)
    total = plan.total_tokens
    qkv = make.rows((case["layers"], total, s.qkv_width))
    out = torch.zeros((case["layers"], total, s.n_q * s.head_dim), dtype=torch.float16, device="cuda")
    scratch = torch.empty(paged.verify_scratch_floats(plan.n_seq, plan.max_tokens_per_seq, s.n_q, s.n_kv,
                                                      s.head_dim, plan.max_len),
                          dtype=torch.float32, device="cuda")
    table, norm = decode.RopeTable(max_len, s.head_dim, s.theta), make.norm(s)

    def step():
        for i, c in enumerate(caches):
            paged.rope_cache(qkv[i], c, table, s.n_q, pos0, cu, total, norm)
            paged.attn_verify(qkv[i], c, out[i], scratch, s.n_q, pos0, cu, total,
                              plan.max_tokens_per_seq, plan.max_len)

    return {"case": case, "step": step, "keep": kv,
            "results": (out, qkv, [c.k for c in caches], [c.v for c in caches])}


def _project(kind, w, x, bias, y, in_f, out_f, n, accumulate):
    (chunk.gemm_fp16 if kind == "fp16" else chunk.gemm_int4_hier)(*w, x, bias, y, in_f, out_f, n, accumulate)


def _prepare_proj(case, s, make):
    kind, layers, n, hid, att = case["weights"], case["layers"], case["n"], HIDDEN[s.name], s.n_q * s.head_dim
    into = [make.weights(kind, hid, s.qkv_width) for _ in range(layers)]
    back = [make.weights(kind, att, hid) for _ in range(layers)]
    # q, k and v have a bias in two of the three models
    bias = [None if s.name == "qwen3-8b" else make.normal((s.qkv_width,)) for _ in range(layers)]
    x, a = make.normal((n, hid)), make.normal((n, att))
    qkv = torch.zeros((layers, n, s.qkv_width), dtype=torch.float32, device="cuda")
    residual = make.rows((n, hid))

    def step():
        for i in range(layers):
            _project(kind, into[i], x, bias[i], qkv[i], hid, s.qkv_width, n, False)
            _project(kind, back[i], a, None, residual, att, hid, n, True)

    return {"case": case, "step": step, "results": (qkv, residual)}


def _prepare_block(case, s, make):
    kind, n_seq, n, hid, att = case["weights"], case["n_seq"], case["n"], HIDDEN[s.name], s.n_q * s.head_dim
    layers, tokens = case["layers"], n_seq * n
    into = [make.weights(kind, hid, s.qkv_width) for _ in range(layers)]
    back = [make.weights(kind, att, hid) for _ in range(layers)]
    caches = [_batch_cache(case, s, make) for _ in range(layers)]
    starts, norm = _starts(case), make.norm(s)
    table = decode.RopeTable(case["max_seq"], s.head_dim, s.theta)
    x, residual = make.normal((tokens, hid)), make.rows((tokens, hid))
    q16 = torch.zeros((tokens, att), dtype=torch.float16, device="cuda")
    out = torch.zeros((layers, tokens, att), dtype=torch.float16, device="cuda")
    project = chunk.qkv_rope_append_batch if kind == "fp16" else chunk.qkv_int4_rope_append_batch

    def step():
        for i in range(layers):
            project(*into[i], x, None, q16, caches[i], table, s.n_q, starts, n, norm)
            chunk.attn_batch_q16(q16, caches[i], out[i], s.n_q, starts, n)
            _project(kind, back[i], out[i], None, residual, att, hid, tokens, True)

    return {"case": case, "step": step,
            "results": (out, q16, residual, [c.k for c in caches], [c.v for c in caches])}


def run(state):
    state["step"]()
    return state["results"]


# ------------------------------------------------------------------- what it must move

def _append_bytes(s, tokens, cache_bytes):
    """qkv rows read, q rows written back, k and v rows written."""
    return tokens * ((s.qkv_width + s.n_q * s.head_dim) * 4 + 2 * s.n_kv * s.head_dim * cache_bytes)


def _attn_bytes(s, tokens, rows, cache_bytes, q_bytes=4):
    """K and V rows once, q rows read, fp16 rows written."""
    return 2 * s.n_kv * rows * s.head_dim * cache_bytes + tokens * s.n_q * s.head_dim * (q_bytes + 2)


def _weight_bytes(kind, in_f, out_f):
    return in_f * out_f * 2 if kind == "fp16" else in_f * out_f // 32 * 17 + out_f * 4


def _proj_work(s, kind, n):
    """Bytes and operations of a layer's two projections, inputs and outputs as they are."""
    hid, att = HIDDEN[s.name], s.n_q * s.head_dim
    nbytes = _weight_bytes(kind, hid, s.qkv_width) + _weight_bytes(kind, att, hid)
    nbytes += n * (hid * 2 + s.qkv_width * 4 + att * 2 + hid * 8)       # the residual is read and written
    return nbytes, 2 * n * hid * (s.qkv_width + att)


def work(case):
    s, kind = SHAPES[case["shape"]], case["kind"]
    flops = nbytes = 0
    if kind == "decode":
        width = 1 if case["cache"] == "e4m3" else 2
        nbytes = case["layers"] * (_append_bytes(s, 1, width) + _attn_bytes(s, 1, case["rows"], width))
        flops = case["layers"] * workloads.prefill_flops(s.n_q, s.head_dim, case["rows"] - 1, 1)
    elif kind in ("chunk", "batch"):
        n, times = case["n"], case["layers"] if kind == "chunk" else case["n_seq"]
        for j in range(case["steps"]):
            pos0 = case["start"] + j * n
            nbytes += times * (_append_bytes(s, n, 2) + _attn_bytes(s, n, pos0 + n, 2))
            flops += times * workloads.prefill_flops(s.n_q, s.head_dim, pos0, n)
    elif kind == "paged":
        for length, n in zip(*_paged_step(case)):
            nbytes += case["layers"] * (_append_bytes(s, n, 2) + _attn_bytes(s, n, length + n, 2))
            flops += case["layers"] * workloads.prefill_flops(s.n_q, s.head_dim, length, n)
    elif kind == "proj":
        b, f = _proj_work(s, case["weights"], case["n"])
        nbytes, flops = case["layers"] * b, case["layers"] * f
    else:
        n, n_seq = case["n"], case["n_seq"]
        tokens = n_seq * n
        b, f = _proj_work(s, case["weights"], tokens)
        b += tokens * (2 * s.n_q * s.head_dim - 4 * s.qkv_width)        # fp16 q rows leave instead of qkv
        b += tokens * 2 * s.n_kv * s.head_dim * 2
        b += n_seq * _attn_bytes(s, n, case["start"] + n, 2, q_bytes=2)
        f += n_seq * workloads.prefill_flops(s.n_q, s.head_dim, case["start"], n)
        nbytes, flops = case["layers"] * b, case["layers"] * f
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times the distance from the same step in 64 bits on the same inputs:
    attention 3.2e-4 to 3.7e-4 (fp16 probabilities and results), the fp16 projections 3.0e-6
    (fp32 sums), the int4 ones 2.0e-4 (weights rounded to fp16 once)."""
    if case["kind"] == "proj":
        return {"rel": 8e-4 if case["weights"] == "int4" else 1.2e-5}
    if case["kind"] == "decode" and case["cache"] == "e4m3":
        # an appended key byte may be the neighbouring one (fp32 rotation)
        return {"rel": 1.5e-3, "differ": 2e-4}
    return {"rel": 1.5e-3}
