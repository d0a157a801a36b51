"""vfkv_decode_token with several layers in a launch: the same rows and outputs as a decode step per layer."""
import numpy as np
import pytest

import vulkanforge_b200 as vf
from util import kv_values, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,scaled,hq,hkv,d,n_layers,lens,windows,n_splits", [
    ("F8", False, 32, 8, 128, 1, [300], None, 0),
    ("F8", False, 8, 1, 128, 70, [130], None, 0),                       # more layers than one launch carries
    ("F8", False, 16, 8, 128, 7, [257, 1, 64], [64, 0, 64, 100, 0, 64, 0], 0),   # windows: a launch for each
    ("F16", False, 16, 8, 256, 5, [500, 33], [128, 128, 128, 128, 0], 3),
    ("F16", False, 4, 2, 64, 3, [2000], None, 64),                      # more splits than the workspace has room for
    ("F32", False, 8, 2, 128, 6, [700, 65], [0, 50, 0, 50, 0, 50], 0),  # CUDA-core kernels: append, split, merge
    ("F32", False, 16, 2, 512, 4, [300, 20], None, 5),
    ("F8", True, 32, 8, 128, 5, [400, 31, 129], None, 0),
])
@pytest.mark.parametrize("slots", [False, True])
def test_layers_of_a_token_share_launches(ctx, dtype, scaled, hq, hkv, d, n_layers, lens, windows, n_splits, slots):
    import torch
    n, longest = len(lens), max(lens)
    rng = np.random.default_rng(n_layers * 100 + longest)
    gen = torch.Generator(device="cuda").manual_seed(longest)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(n_layers, hkv, d, longest + 3, n_slots=n + 1, scale_mode=int(scaled)),
                       vf.KvDtype[dtype])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, max_batch=n, n_splits=n_splits)
    ids = list(range(n, 0, -1)) if slots else list(range(n))
    try:
        for layer in range(n_layers):
            for i, length in enumerate(lens):
                kv = torch.randn(2, length, hkv, d, device="cuda", generator=gen)
                fwd.b_step_kv_write(layer, kv[0], kv[1], length, 0, ids[i])
        q = torch.randn(n_layers, n, hq, d, device="cuda", generator=gen)
        k = to_dev(kv_values(rng, (n_layers, n, hkv, d)))
        v = to_dev(kv_values(rng, (n_layers, n, hkv, d)))
        pos = to_dev(np.array([x - 1 for x in lens], np.uint32))
        d_ids = to_dev(np.array(ids, np.uint32)) if slots else None
        row = cache.row_bytes(0)

        def state():
            torch.cuda.synchronize()
            L, out = ctx._lib, np.empty((2, cache.bytes_per_buffer()), np.uint8)
            for o, a in zip(out, (cache.k_buffer, cache.v_buffer)):
                ctx.check(L.vfkv_memcpy_d2h(ctx.handle, o.ctypes.data, a, o.nbytes, None))
            ctx.check(L.vfkv_stream_synchronize(ctx.handle, None))
            return [out[:, cache.slot_offset_bytes(l, s) + (x - 1) * row:][:, :row].copy()
                    for l in range(n_layers) for s, x in zip(ids, lens)]

        per_layer, together = torch.zeros_like(q), torch.zeros_like(q)
        w_of = lambda l: windows[l] if windows else 0
        for layer in range(n_layers):
            fwd.sliding_layers, fwd.sliding_window = ({layer}, w_of(layer)) if w_of(layer) else (set(), 0)
            fwd.decode_step(layer, q[layer], k[layer], v[layer], per_layer[layer], d_ids, pos, n, longest)
        want = state()
        for layer in range(n_layers):                      # other rows in the token's place, to be overwritten again
            for i, length in enumerate(lens):
                z = torch.zeros(2, 1, hkv, d, device="cuda")
                fwd.b_step_kv_write(layer, z[0], z[1], 1, length - 1, ids[i])
        kernels = ctx.kernel_count()
        import ctypes as C
        arr = (C.c_uint32 * n_layers)(*windows) if windows else None
        ctx.check(ctx._lib.vfkv_decode_token(cache.handle, fwd.workspace.handle, q.data_ptr(), k.data_ptr(), v.data_ptr(),
                                             together.data_ptr(), hq, None if d_ids is None else d_ids.data_ptr(),
                                             pos.data_ptr(), n, longest, C.cast(arr, C.c_void_p) if windows else None,
                                             fwd.attn_scale, 0.0, n_splits, None))
        got = state()
        ctx.poll()
        launches = len(set(windows)) if windows else -(-n_layers // 64)
        assert ctx.kernel_count() - kernels <= 3 * launches
        assert all(np.array_equal(a, b) for a, b in zip(want, got))
        scale = float(per_layer.abs().max())
        assert float((together - per_layer).abs().max()) < 2e-5 * max(1.0, scale)
    finally:
        fwd.workspace.destroy()
        cache.destroy()


@pytest.mark.parametrize("n_layers,n,pinned", [(3, 2, "all"), (40, 8, "all"), (3, 2, "none"), (40, 8, "inputs"), (3, 2, "output")])
def test_host_token_pinned_buffers_and_replays(ctx, n_layers, n, pinned):
    """vfkv_decode_token_host by every way its buffers can travel (one kernel, groups of layers, pageable),
    called again with the same buffers (a recording) and alternating between two sets of them."""
    import torch
    hq, hkv, d, length = 32, 8, 128, 200
    gen = torch.Generator().manual_seed(n_layers)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(n_layers, hkv, d, 256, n_slots=n), vf.KvDtype.F16)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, max_batch=n)
    ref = vf.CudaForward(ctx, cache, n_heads=hq, max_batch=n)
    stream = torch.cuda.Stream()
    try:
        cache.zero_fill()
        for layer in range(n_layers):
            for slot in range(n):
                kv = torch.randn(2, length, hkv, d, generator=gen).cuda()
                fwd.b_step_kv_write(layer, kv[0], kv[1], length, 0, slot)
        torch.cuda.synchronize()
        fwd.stream = stream.cuda_stream
        host = lambda x, when: x.pin_memory() if pinned in ("all", when) else x
        sets = [[host(torch.randn(n_layers, n, h, d, generator=gen), "inputs") for h in (hq, hkv, hkv)] +
                [host(torch.zeros(n_layers, n, hq, d), "output")] for _ in range(2)]
        for step, which in enumerate((0, 0, 0, 1, 1, 0, 1)):
            q, k, v, out = sets[which]
            q.normal_(generator=gen)
            out.fill_(7.0)
            pos = np.array([length + step - 3 * i for i in range(n)], np.uint32)
            ids = np.arange(n, dtype=np.uint32)[::-1].copy() if step % 2 else None
            fwd.decode_token_host(q, k, v, out, pos, n, ids)
            want = torch.zeros(n_layers, n, hq, d, device="cuda")
            ref.decode_token(q.cuda(), k.cuda(), v.cuda(), want, None if ids is None else to_dev(ids), to_dev(pos), n, 256)
            torch.cuda.synchronize()
            assert float((want.cpu() - out).abs().max()) < 1e-5
        ctx.poll()
    finally:
        fwd.stream = None
        fwd.workspace.destroy()
        ref.workspace.destroy()
        cache.destroy()


@pytest.mark.parametrize("dtype,hq,hkv,d,layers,L", [
    ("F8", 32, 8, 128, 20, 8192),          # heads on the N side: one CTA for each of 160 groups
    ("F16", 64, 8, 128, 20, 8192),         # heads on the M side
    ("F16", 32, 4, 256, 12, 16384),
    ("F16", 16, 2, 512, 4, 20000),         # attn_wide.cu
])
def test_long_sums_keep_their_accuracy(ctx, dtype, hq, hkv, d, layers, L):
    """Layers that share a launch leave a warp a long line of positions.  What its sums lose there (to the tensor cores'
    cutting off: 2^-24 of the sum for each product) must not exceed what f32 sums lose: results within 2^-20."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(d)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(layers, hkv, d, L), vf.KvDtype[dtype])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    try:
        rows = torch.randn(layers, 2, L, hkv, d, device="cuda", generator=gen)
        rows = rows.to(torch.float8_e4m3fn).float() if dtype == "F8" else rows.half().float()
        for i in range(layers):
            fwd.b_step_kv_write(i, rows[i, 0, :L - 1], rows[i, 1, :L - 1], L - 1, 0)
        q, out = torch.randn(layers, 1, hq, d, device="cuda", generator=gen), torch.zeros(layers, 1, hq, d, device="cuda")
        new = rows[:, :, L - 1].contiguous()
        fwd.decode_token(q, new[:, 0].contiguous(), new[:, 1].contiguous(), out, None,
                         torch.tensor([L - 1], dtype=torch.int32, device="cuda"), 1, L)
        worst = 0.0
        for i in range(layers):
            k, v = rows[i, 0].double(), rows[i, 1].double()
            s = torch.einsum("hgd,lhd->hgl", q[i, 0].double().view(hkv, hq // hkv, d), k) / d ** 0.5
            want = torch.einsum("hgl,lhd->hgd", s.softmax(-1), v).reshape(hq, d)
            worst = max(worst, float((out[i, 0].double() - want).norm() / want.norm()))
        assert worst < 2.0 ** -20
    finally:
        fwd.workspace.destroy()
        cache.destroy()


def test_phase_trace_stays_in_its_buffer(ctx):
    """A ring of one block for each layer's launch (16 x 8 bytes a CTA): decode_token fills it and writes nothing behind it."""
    import torch
    hq, hkv, d, layers, L, splits = 32, 8, 128, 6, 4096, 4
    own = vf.Context(0)
    cache = vf.KvCache(own, vf.KvCacheConfig(layers, hkv, d, L), vf.KvDtype.F8)
    fwd = vf.CudaForward(own, cache, n_heads=hq, n_splits=splits)
    try:
        cache.zero_fill()
        words = layers * hkv * splits * 16
        ring = torch.zeros(words + 65536, dtype=torch.int64, device="cuda")
        q, out = (torch.zeros(layers, 1, hq, d, device="cuda") for _ in range(2))
        kv = torch.zeros(2, layers, 1, hkv, d, device="cuda")
        own.check(own._lib.vfkv_ctx_set_trace_buffer(own.handle, ring.data_ptr()))
        own.check(own._lib.vfkv_ctx_set_trace_ring(own.handle, layers))
        for _ in range(3):
            fwd.decode_token(q, kv[0], kv[1], out, None, torch.tensor([L - 1], dtype=torch.int32, device="cuda"), 1, L)
        torch.cuda.synchronize()
        assert (ring[:words].view(-1, 16)[:, 0] != 0).all() and not ring[words:].any()
    finally:
        own.check(own._lib.vfkv_ctx_set_trace_buffer(own.handle, None))
        fwd.workspace.destroy()
        cache.destroy()
        own.destroy()


def test_recorded_token_follows_the_scale_planes(ctx):
    """A cache made anew where another one's K and V lay, with its scales elsewhere: the token recorded for the old one
    (same buffers, same sizes) is not the new one's."""
    import ctypes as C
    import torch
    hq, hkv, d, layers, L = 16, 8, 128, 2, 4096
    gen = torch.Generator(device="cuda").manual_seed(9)
    rows = torch.randn(layers, 2, L, hkv, d, device="cuda", generator=gen)
    q, out = (torch.zeros(layers, 1, hq, d).pin_memory() for _ in range(2))
    q.copy_(torch.randn(layers, 1, hq, d))
    new = rows[:, :, L - 1].cpu()
    k, v = new[:, 0].contiguous().pin_memory(), new[:, 1].contiguous().pin_memory()
    pos = np.array([L - 1], np.uint32)
    ws, fillers, planes = None, [], layers * L * hkv * 4
    stream = torch.cuda.Stream()
    try:
        for again in range(2):
            cache = vf.KvCache(ctx, vf.KvCacheConfig(layers, hkv, d, L, scale_mode=1), vf.KvDtype.F8)
            fwd = vf.CudaForward(ctx, cache, n_heads=hq, workspace=ws)
            ws, fwd.stream = fwd.workspace, stream.cuda_stream
            scale = 1.0 + 3.0 * again
            for i in range(layers):
                fwd.b_step_kv_write(i, rows[i, 0, :L - 1] * scale, rows[i, 1, :L - 1] * scale, L - 1, 0)
            for _ in range(3):                             # remembered, recorded, replayed
                fwd.decode_token_host(q, k, v, out, pos, 1)
            want = torch.zeros(layers, 1, hq, d, device="cuda")
            dq, dk, dv = q.cuda(), k.cuda(), v.cuda()
            for i in range(layers):
                fwd.decode_step(i, dq[i], dk[i], dv[i], want[i], None, to_dev(pos), 1, L)
            torch.cuda.synchronize()
            assert float((out - want.cpu()).abs().max()) < 1e-5 * max(1.0, float(want.abs().max()))
            cache.destroy()
            for _ in range(2):                             # where the scales lay
                p = C.c_void_p()
                ctx.check(ctx._lib.vfkv_malloc(ctx.handle, planes, C.byref(p)))
                fillers.append(p)
    finally:
        for p in fillers:
            ctx.check(ctx._lib.vfkv_free(ctx.handle, p))
        ws.destroy()


def test_kernel_count_of_a_host_token(ctx):
    """From pinned buffers: one kernel fetches the inputs, one does all layers, recorded or not."""
    import torch
    hq, hkv, d, layers = 16, 8, 128, 3
    cache = vf.KvCache(ctx, vf.KvCacheConfig(layers, hkv, d, 64), vf.KvDtype.F8)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    stream = torch.cuda.Stream()
    try:
        fwd.stream = stream.cuda_stream
        q, out = (torch.zeros(layers, 1, hq, d).pin_memory() for _ in range(2))
        k, v = (torch.zeros(layers, 1, hkv, d).pin_memory() for _ in range(2))
        for p in range(4):
            kernels, launches = ctx.kernel_count(), ctx.launch_count()
            fwd.decode_token_host(q, k, v, out, np.array([p], np.uint32), 1)
            assert (ctx.kernel_count() - kernels, ctx.launch_count() - launches) == (2, layers)
    finally:
        fwd.workspace.destroy()
        cache.destroy()


def test_host_buffer_with_an_unregistered_page_is_not_pinned(ctx):
    """Four pages of Q, the third not registered: no kernel reads that buffer, whatever its two ends are."""
    import mmap
    import torch
    hq, hkv, d, layers, page = 16, 8, 128, 2, mmap.PAGESIZE
    cache = vf.KvCache(ctx, vf.KvCacheConfig(layers, hkv, d, 64), vf.KvDtype.F8)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    stream, cudart = torch.cuda.Stream(), torch.cuda.cudart()
    memory = mmap.mmap(-1, layers * hq * d * 4)
    q = np.frombuffer(memory, np.float32).reshape(layers, 1, hq, d)
    at = q.ctypes.data
    parts = [(at, 2 * page), (at + 3 * page, q.nbytes - 3 * page)]
    q[:] = np.random.default_rng(1).standard_normal(q.shape, dtype=np.float32)
    out = torch.zeros(layers, 1, hq, d).pin_memory()
    k, v = (torch.randn(layers, 1, hkv, d).pin_memory() for _ in range(2))
    try:
        for p, n in parts:
            assert int(cudart.cudaHostRegister(p, n, 0)) == 0
        fwd.stream = stream.cuda_stream
        kernels = ctx.kernel_count()
        try:
            fwd.decode_token_host(q, k, v, out, np.array([0], np.uint32), 1)
        except vf.VfkvError:                               # the runtime may refuse to copy such a range
            return
        assert ctx.kernel_count() - kernels == 1
        want = v.to(torch.float8_e4m3fn).float().repeat_interleave(hq // hkv, 2)     # one position: its V
        assert float((out - want).abs().max()) < 1e-5 * float(want.abs().max())
    finally:
        for p, _ in parts:
            cudart.cudaHostUnregister(p)
        fwd.workspace.destroy()
        cache.destroy()
