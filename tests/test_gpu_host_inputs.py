"""decode_token_host from pinned buffers of more whole sequences than the GPU holds CTAs of at a time: the launch reads Q, the new
rows, positions and slots out of host memory itself; up to that many, a kernel fetches them first.  The same bits as decode_token
from device memory, which makes the same launches."""
import numpy as np
import pytest

import vulkanforge_b200 as vf
from util import kv_values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,scaled,hq,hkv,d,n_layers,lens,capacity,window,softcap,slots,kernels", [
    ("F8", False, 32, 8, 128, 19, [600, 70, 33], 1024, 0, 0.0, True, 1),          # 456 pairs, four warps a CTA
    ("F8", False, 64, 8, 128, 7, [1, 200, 64, 90, 5, 33, 7], 1024, 0, 30.0, False, 1),       # 3.5 MB; eight q-heads: 4 KB of Q
    ("F8", True, 32, 8, 128, 56, [600], 1024, 0, 0.0, False, 1),
    ("F8", False, 32, 8, 128, 26, [60, 31, 5], 256, 0, 0.0, False, 1),            # at most eight tiles: a warp a sequence
    ("F16", False, 16, 8, 256, 38, [40, 17, 100], 1024, 50, 0.0, True, 2),        # a window in half of the layers: a launch each
    ("F16", False, 16, 1, 128, 48, [90, 20, 1, 64, 33, 17, 16, 100, 5, 128], 128, 0, 0.0, False, 1),      # the same; sixteen q-heads: 8 KB of Q
    ("F16", False, 8, 8, 64, 38, [128, 100], 256, 0, 50.0, False, 1),             # 608 pairs, however short
    ("F16", False, 32, 8, 128, 38, [600], 1024, 0, 0.0, False, 1),                # 304 of 300 KB
    ("F8", False, 32, 8, 128, 36, [70], 1024, 0, 0.0, False, 2),                  # 288 pairs: the inputs are fetched first
    ("F16", False, 32, 8, 128, 37, [600], 1024, 0, 0.0, False, 2),                # the most that they are for: 296 of 300 KB,
    ("F16", False, 40, 8, 128, 38, [600], 1024, 0, 0.0, False, 2),                # 304 where groups have five heads,
    ("F8", False, 32, 8, 128, 55, [600], 1024, 0, 0.0, True, 2),                  # 440 of 150 KB,
    ("F16", False, 8, 8, 64, 37, [128, 100], 256, 0, 0.0, False, 2),              # 592 of less
    ("F16", False, 8, 8, 64, 50, [128, 90], 256, 50, 0.0, True, 3),               # 800, but 400 in each of two launches
])
def test_inputs_straight_from_the_host(ctx, dtype, scaled, hq, hkv, d, n_layers, lens, capacity, window, softcap, slots, kernels):
    import torch
    n, longest = len(lens), max(lens)
    gen = torch.Generator(device="cuda").manual_seed(longest + d)
    rng = np.random.default_rng(longest)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(n_layers, hkv, d, capacity, n_slots=n + 1, scale_mode=int(scaled)), vf.KvDtype[dtype])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, max_batch=n, softcap=softcap, sliding_window=window,
                         sliding_layers=range(n_layers // 2) if window else (), n_splits=1)
    ids = list(range(n, 0, -1)) if slots else list(range(n))
    stream = torch.cuda.Stream()
    try:
        for layer in range(n_layers):
            for i, length in enumerate(lens):
                kv = torch.randn(2, length, hkv, d, device="cuda", generator=gen)
                fwd.b_step_kv_write(layer, kv[0], kv[1], length, 0, ids[i])
        torch.cuda.synchronize()
        q = torch.randn(n_layers, n, hq, d).pin_memory()
        k, v = (torch.from_numpy(kv_values(rng, (n_layers, n, hkv, d))).pin_memory() for _ in range(2))
        out = torch.full((n_layers, n, hq, d), float("nan")).pin_memory()
        pos = np.array([x - 1 for x in lens], np.uint32)
        h_ids = np.array(ids, np.uint32) if slots else None

        def state():
            torch.cuda.synchronize()
            b = np.empty((2, cache.bytes_per_buffer()), np.uint8)
            for o, a in zip(b, (cache.k_buffer, cache.v_buffer)):
                ctx.check(ctx._lib.vfkv_memcpy_d2h(ctx.handle, o.ctypes.data, a, o.nbytes, None))
            ctx.check(ctx._lib.vfkv_stream_synchronize(ctx.handle, None))
            return b

        fwd.stream = stream.cuda_stream
        before = ctx.kernel_count()
        fwd.decode_token_host(q, k, v, out, pos, n, h_ids)
        assert ctx.kernel_count() - before == kernels
        ctx.poll()
        got = state()
        fwd.stream = None
        d_out = torch.zeros(n_layers, n, hq, d, device="cuda")
        fwd.decode_token(q.cuda(), k.cuda(), v.cuda(), d_out, torch.from_numpy(h_ids.view(np.int32)).cuda() if slots else None,
                         torch.from_numpy(pos.view(np.int32)).cuda(), n, capacity)
        assert (state() == got).all()
        assert torch.equal(out, d_out.cpu())
    finally:
        fwd.workspace.destroy()
        cache.destroy()
