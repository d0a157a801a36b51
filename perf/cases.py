"""The work a host has this library do, as cases that can be timed.

A case names one pass through the public entry points (``CudaForward`` over a ``KvCache``) and its
sizes.  Five kinds of pass:

  token    every layer's KvWrite + attention for one token of each sequence, one call, device buffers
           (``decode_token``): decoding, the bulk of what a server does
  step     the same layer by layer with the executor's two calls (``step_kv_write``,
           ``step_attention``): a single-stream forward loop that interleaves its own kernels
  host     ``decode_token_host``: the same token from pinned host buffers, waited for
  prefill  one layer of a prompt chunk: RoPE on Q, RoPE + append of K and V, causal attention of the
           chunk over everything cached so far
  chunk    plain append of a prompt chunk and, for FP8 caches, the F16 read-out of the cached rows that
           a host-side attention kernel would use

Shapes are those of the repository's workloads and tests (q-heads / kv-heads / head_dim 32/8/128,
64/8/128, 16/8/256, ...); K and V are N(0, 1), with one element in a hundred twenty times larger for
FP8 caches.
"""
import math
import random

import numpy as np
import torch

import vulkanforge_b200 as vf

ROPE_BASE = 500000.0
ELEMENT = {"F32": 4, "F16": 2, "F8": 1}


def _case(name, kind, dtype, heads, ctx, *, seqs=1, layers=1, scaled=False, chunk=0, shortest=0, window=0,
          sliding=0, softcap=0.0):
    """ctx: positions attended over by the last query, its own included.  shortest: sequence lengths are
    spread over [shortest, ctx].  The first ``sliding`` layers see only ``window`` positions."""
    c = {"kind": kind, "dtype": dtype, "scaled": scaled, "q_heads": heads[0], "kv_heads": heads[1],
         "head_dim": heads[2], "layers": layers, "seqs": seqs, "ctx": ctx, "shortest": shortest or ctx,
         "chunk": chunk, "window": window, "sliding": sliding, "softcap": softcap}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest: one layer of a single short chat, F16 cache; launches and host calls are all of it
        _case("step_f16_b1_2048", "step", "F16", (32, 8, 128), 2048),
        # one user's token through a whole 36-layer model, FP8 cache
        _case("token_fp8_b1_8192", "token", "F8", (32, 8, 128), 8192, layers=36),
        # a server's batch: 64 sequences of very different lengths
        _case("token_fp8_b64_ragged", "token", "F8", (32, 8, 128), 16384, seqs=64, layers=2, shortest=512),
        # wide heads, F16, five sliding-window layers to one global layer, soft-capped scores
        _case("token_f16_d256_b8_32768", "token", "F16", (16, 8, 256), 32768, seqs=8, layers=6, window=1024, sliding=5,
              softcap=50.0),
        # one very long document, eight q-heads to a kv-head
        _case("token_fp8_g8_131072", "token", "F8", (64, 8, 128), 131072, layers=8),
        # FP8 with a scale for each token and head, a handful of sequences of odd length
        _case("token_fp8_scaled_b8_4099", "token", "F8", (32, 8, 128), 4099, seqs=8, layers=4, scaled=True,
              shortest=2001),
        # the end-to-end boundary of a host that keeps its activations in host memory
        _case("host_fp8_b1_8192", "host", "F8", (32, 8, 128), 8192, layers=36),
        # a large chunk late in a long prompt: the largest contraction
        _case("prefill_fp8_2048_of_16384", "prefill", "F8", (32, 8, 128), 16384, chunk=2048),
        # the ragged last chunk of an ordinary prompt, F16
        _case("prefill_f16_333_of_1333", "prefill", "F16", (32, 8, 128), 1333, chunk=333),
        # a chunk of a sliding-window layer with wide heads and soft-capped scores
        _case("prefill_f16_d256_1024_of_5120", "prefill", "F16", (16, 8, 256), 5120, chunk=1024, window=1024, sliding=1,
              softcap=50.0),
        # the full-precision cache: a short prompt
        _case("prefill_f32_200_of_700", "prefill", "F32", (32, 8, 128), 700, chunk=200),
        # a 512-token chunk into an FP8 cache of four layers and the F16 read-out of what it holds by then
        _case("chunk_fp8_512_of_8192", "chunk", "F8", (32, 8, 128), 8192, layers=4, chunk=512),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choices(["token", "step", "host", "prefill", "chunk"], [40, 12, 8, 30, 10])[0]
    dtype, scaled = rng.choices([("F8", False), ("F16", False), ("F8", True), ("F32", False)], [45, 35, 10, 10])[0]
    if kind == "prefill":
        heads = rng.choices([(32, 8, 128), (64, 8, 128), (16, 8, 256), (8, 8, 64)], [5, 2, 2, 1])[0]
    else:
        heads = rng.choices([(32, 8, 128), (64, 8, 128), (16, 8, 256), (8, 8, 64), (40, 8, 128), (8, 1, 128), (32, 2, 128),
                             (16, 2, 512)], [8, 4, 4, 1, 1, 1, 1, 1])[0]
    wide = dtype == "F32" or scaled or heads[2] == 512     # what full precision, scales or very wide heads are used for is smaller
    softcap = rng.choice([30.0, 50.0]) if rng.random() < 0.2 else 0.0
    row = 2 * heads[1] * heads[2] * ELEMENT[dtype]         # K and V of one position of one layer
    if kind in ("token", "step", "host"):
        most = (256 << 20) if wide else (2 << 30)          # bytes of K and V read in a pass
        layers = rng.choice([1, 2, 4, 8, 16, 32] if kind != "host" else [4, 9, 16, 32])
        seqs = 1 if kind == "step" else _log_int(rng, 1, 64)
        ctx = _log_int(rng, 16, max(64, min(131072, most // (layers * seqs * row))))
        shortest = _log_int(rng, max(1, ctx // 32), ctx) if seqs > 1 and rng.random() < 0.6 else 0
        sliding = layers * 5 // 6 if ctx > 1100 and rng.random() < 0.25 else 0
        return _case(None, kind, dtype, heads, ctx, seqs=seqs, layers=layers, scaled=scaled, shortest=shortest,
                     window=1024 if sliding else 0, sliding=sliding, softcap=softcap)
    if kind == "chunk":
        ctx = _log_int(rng, 32, 16384)
        return _case(None, kind, dtype, heads, ctx, layers=rng.choice([4, 8, 16]), scaled=scaled,
                     chunk=_log_int(rng, 16, min(ctx, 2048)))
    flops = 6e9 if wide else 6e10 if heads[2] != 128 else 4e11     # of a pass, as if nothing were masked
    chunk = _log_int(rng, 16, 512 if wide else 2048)
    ctx = _log_int(rng, chunk, max(chunk, min(65536, int(flops / (4 * heads[0] * heads[2] * chunk)))))
    window = 1024 if ctx > 1100 and rng.random() < 0.25 else 0
    return _case(None, kind, dtype, heads, ctx, scaled=scaled, chunk=chunk, window=window, sliding=1 if window else 0,
                 softcap=softcap)


def _lengths(case):
    """Sequence lengths, the longest first; a property of the case, not of the seed."""
    rng = random.Random(case["ctx"] * 64 + case["seqs"])
    return [case["ctx"]] + [rng.randint(case["shortest"], case["ctx"]) for _ in range(case["seqs"] - 1)]


_context = None


def _ctx():
    """One library context for the process, as a program has.  Dependent-launch mode 2: what precedes an
    attention call on the stream (a projection, another layer) writes neither its rows nor its positions."""
    global _context
    if _context is None:
        _context = vf.Context(0)
        _context.set_dependent_launch(2)
    return _context


class _Handles:
    """Cache and workspace, given back with the last object that refers to them."""

    def __init__(self, cache, fwd):
        self.owned = (fwd.workspace, cache)

    def __del__(self):
        torch.cuda.synchronize()
        for handle in self.owned:
            handle.destroy()


class _Memory:
    """Device memory of the cache for ``torch.as_tensor``: 64-bit words, no copy; the tensor keeps the cache."""

    def __init__(self, handles, address, n_bytes):
        self.handles = handles
        self.__cuda_array_interface__ = {"shape": (n_bytes // 8,), "typestr": "<i8", "data": (address, False), "version": 2}


class _State:
    """What a program keeps between calls."""

    def __init__(self, case):
        self.case = case
        c = case
        self.lens = _lengths(c)
        capacity = -(-c["ctx"] // 256) * 256
        self.cache = vf.KvCache(_ctx(), vf.KvCacheConfig(c["layers"], c["kv_heads"], c["head_dim"], capacity,
                                                         n_slots=c["seqs"], scale_mode=int(c["scaled"])),
                                vf.KvDtype[c["dtype"]])
        self.fwd = vf.CudaForward(_ctx(), self.cache, n_heads=c["q_heads"], max_batch=c["seqs"], softcap=c["softcap"],
                                  sliding_window=c["window"], sliding_layers=range(c["sliding"]))
        self.handles = _Handles(self.cache, self.fwd)
        n = self.cache.bytes_per_buffer()
        self.memory = [torch.as_tensor(_Memory(self.handles, p, n), device="cuda") for p in (self.cache.k_buffer, self.cache.v_buffer)]
        if c["scaled"]:
            planes = c["layers"] * c["seqs"] * capacity * c["kv_heads"] * 4
            self.memory += [torch.as_tensor(_Memory(self.handles, p, planes), device="cuda").view(torch.float32)
                            for p in (self.cache.k_scales, self.cache.v_scales)]


def _values(gen, case, *shape):
    x = torch.randn(*shape, device="cuda", generator=gen)
    if case["dtype"] == "F8":
        x = torch.where(torch.rand(*shape, device="cuda", generator=gen) < 0.01, x * 20.0, x)
    return x


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = _State(c)
    s.cache.zero_fill()
    hq, hkv, d, n, layers = c["q_heads"], c["kv_heads"], c["head_dim"], c["seqs"], c["layers"]
    new = c["chunk"] or 1                                  # tokens that the pass itself stores, of each sequence
    for layer in range(layers):                            # the tokens before it
        for slot, length in enumerate(s.lens):
            for p in range(0, length - new, 32768):
                m = min(32768, length - new - p)
                kv = _values(gen, c, 2, m, hkv, d)
                s.fwd.b_step_kv_write(layer, kv[0], kv[1], m, p, slot)
    if c["kind"] in ("token", "step", "host"):
        s.q = torch.randn(layers, n, hq, d, device="cuda", generator=gen)
        s.k, s.v = _values(gen, c, layers, n, hkv, d), _values(gen, c, layers, n, hkv, d)
        s.out = torch.zeros(layers, n, hq, d, device="cuda")
        s.positions = torch.tensor([x - 1 for x in s.lens], dtype=torch.int32, device="cuda")
    elif c["kind"] == "prefill":
        s.q = torch.randn(new, hq, d, device="cuda", generator=gen)
        s.k, s.v = _values(gen, c, new, hkv, d), _values(gen, c, new, hkv, d)
    else:
        s.k, s.v = _values(gen, c, layers, new, hkv, d), _values(gen, c, layers, new, hkv, d)
    if c["kind"] == "host":
        s.q, s.k, s.v, s.out = (t.cpu().pin_memory() for t in (s.q, s.k, s.v, s.out))
        s.positions = np.array([x - 1 for x in s.lens], np.uint32)
        s.stream = torch.cuda.Stream()
        s.fwd.stream = s.stream.cuda_stream
    if c["kind"] == "prefill":
        s.q_rot, s.out = torch.zeros_like(s.q), torch.zeros_like(s.q)
        s.k_rot = torch.zeros_like(s.k) if c["scaled"] else None            # scales are taken from the rotated rows
    if c["kind"] == "chunk" and c["dtype"] == "F8":
        s.read = torch.zeros(layers, 2, c["ctx"] * hkv * d, dtype=torch.float16, device="cuda")
        s.slabs = [(s.cache.k_buffer + s.cache.layer_offset_bytes(i), s.cache.v_buffer + s.cache.layer_offset_bytes(i))
                   for i in range(layers)]
    torch.cuda.synchronize()
    return s


def run(s):
    c, fwd = s.case, s.fwd
    if c["kind"] == "token":
        fwd.decode_token(s.q, s.k, s.v, s.out, None, s.positions, c["seqs"], c["ctx"])
        return {"out": s.out, "cache": s.memory}
    if c["kind"] == "step":
        for layer in range(c["layers"]):
            fwd.step_kv_write(layer, s.k[layer], s.v[layer], c["ctx"] - 1)
            fwd.step_attention(layer, s.q[layer], s.out[layer], c["ctx"] - 1)
        return {"out": s.out, "cache": s.memory}
    if c["kind"] == "host":
        fwd.decode_token_host(s.q, s.k, s.v, s.out, s.positions, c["seqs"])
        return {"out": s.out, "cache": s.memory}
    m, base = c["chunk"], c["ctx"] - c["chunk"]
    if c["kind"] == "prefill":
        fwd.run_rope_neox(s.q, s.q_rot, m, c["q_heads"], c["head_dim"], base, freq_base=ROPE_BASE)
        fwd.rope_kv_write(0, s.k, s.v, m, base, k_rot=s.k_rot, freq_base=ROPE_BASE)
        fwd.b_step_attention(0, s.q_rot, s.out, m, base, exact_window=True)
        return {"out": s.out, "q": s.q_rot, "cache": s.memory}
    for layer in range(c["layers"]):
        fwd.b_step_kv_write(layer, s.k[layer], s.v[layer], m, base)
        if c["dtype"] == "F8":
            for slab, read in zip(s.slabs[layer], s.read[layer]):
                fwd.run_kv_fp8_to_f16(slab, read, c["ctx"] * c["kv_heads"] * c["head_dim"])
    return {"cache": s.memory, "read": s.read if c["dtype"] == "F8" else None}


def work(case):
    c = case
    kv_elems, q_elems = c["kv_heads"] * c["head_dim"], c["q_heads"] * c["head_dim"]
    row = 2 * (kv_elems * ELEMENT[c["dtype"]] + (4 * c["kv_heads"] if c["scaled"] else 0))    # K and V of one position
    lens, new = _lengths(c), c["chunk"] or 1
    stored = new * len(lens) * c["layers"] * (row + 2 * kv_elems * 4)                         # f32 in, cache rows out
    if c["kind"] == "chunk":
        return {"bytes": stored + (c["layers"] * c["ctx"] * 2 * kv_elems * 3 if c["dtype"] == "F8" else 0), "flops": 0}
    rows = pairs = 0                                       # cached positions read, (query, position) pairs
    for layer in range(c["layers"]):
        window = c["window"] if layer < c["sliding"] else 0
        for length in lens:
            rows += min(length, window + new - 1) if window else length
            seen = range(length - new + 1, length + 1)
            pairs += sum(min(x, window) for x in seen) if window else new * (seen[0] + seen[-1]) // 2
    rows -= new * len(lens) * c["layers"]                  # the new rows need not be read back
    moved = q_elems * 4 * new * len(lens) * c["layers"] * (3 if c["kind"] == "prefill" else 2)
    return {"bytes": rows * row + stored + moved, "flops": 4 * q_elems * pairs}


def tolerance(case):
    """Decode keeps 32-bit accuracy (half-precision operands are split into two terms, except for groups
    of more than eight q-heads); the prefill kernels feed Q and P of F8 and F16 caches as half precision.
    Cache bytes are exact."""
    group = case["q_heads"] // case["kv_heads"]
    if case["kind"] == "chunk":
        return "exact"
    if case["dtype"] == "F32" or case["scaled"]:
        return {"rel": 2e-5}                               # 32-bit sums over up to some ten thousand positions
    if case["kind"] == "prefill" or group > 8:
        return {"rel": 2e-3}
    return {"rel": 1e-5}
