"""decode_token_host from pinned buffers where every SM has whole sequences to stream: the launch reads Q, the new rows, positions
and slots out of host memory itself.  The same bits as decode_token from device memory, which makes the same launches."""
import numpy as np
import pytest

import vulkanforge_b200 as vf
from util import kv_values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,scaled,hq,hkv,d,n_layers,lens,window,softcap,slots", [
    ("F8", False, 32, 8, 128, 10, [70, 33], 0, 0.0, True),               # 160 pairs, four warps a CTA
    ("F8", False, 64, 8, 128, 7, [1, 200, 64], 0, 30.0, False),          # eight q-heads a kv-head: 4 KB of Q
    ("F8", True, 32, 8, 128, 19, [300], 0, 0.0, False),
    ("F8", False, 32, 8, 128, 24, [60, 31, 5], 0, 0.0, False),           # a warp a sequence
    ("F16", False, 16, 8, 256, 14, [40, 17, 100], 50, 0.0, True),        # a window in some layers: two launches
    ("F16", False, 16, 1, 128, 33, [90, 20, 1, 64, 33], 0, 0.0, False),  # sixteen q-heads: 8 KB of Q
    ("F16", False, 8, 8, 64, 20, [128], 0, 50.0, False),
])
def test_inputs_straight_from_the_host(ctx, dtype, scaled, hq, hkv, d, n_layers, lens, window, softcap, slots):
    import torch
    n, longest = len(lens), max(lens)
    gen = torch.Generator(device="cuda").manual_seed(longest + d)
    rng = np.random.default_rng(longest)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(n_layers, hkv, d, 1024, n_slots=n + 1, scale_mode=int(scaled)), vf.KvDtype[dtype])
    # half of the layers see a window: each launch still has a CTA for every SM
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
        kernels = ctx.kernel_count()
        fwd.decode_token_host(q, k, v, out, pos, n, h_ids)
        assert ctx.kernel_count() - kernels == (2 if window else 1)
        ctx.poll()
        got = state()
        fwd.stream = None
        d_out = torch.zeros(n_layers, n, hq, d, device="cuda")
        fwd.decode_token(q.cuda(), k.cuda(), v.cuda(), d_out, torch.from_numpy(h_ids.view(np.int32)).cuda() if slots else None,
                         torch.from_numpy(pos.view(np.int32)).cuda(), n, 1024)
        assert (state() == got).all()
        assert torch.equal(out, d_out.cpu())
    finally:
        fwd.workspace.destroy()
        cache.destroy()
