"""Decode shapes outside one tensor-core tile -- more q-heads than it holds, 512-dim heads, 64-dim FP8 rows --
against the CUDA-core kernel, which the oracle tests cover."""
import numpy as np
import pytest

import vulkanforge_b200 as vf
from util import kv_values, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,scaled,hq,hkv,d,lens,window,softcap,n_splits", [
    ("F8", False, 32, 2, 128, [1, 300, 4100], 0, 0.0, 0),
    ("F8", False, 9, 1, 128, [700], 0, 0.0, 3),             # three parts of three heads
    ("F8", False, 22, 2, 256, [33, 257], 100, 30.0, 0),     # eleven parts of one
    ("F8", True, 32, 2, 128, [129, 31], 0, 0.0, 2),
    ("F16", False, 34, 2, 128, [600], 0, 0.0, 0),
    ("F16", False, 24, 1, 64, [65, 64], 0, 50.0, 1),
    # 512-dim heads and 64-dim FP8 rows: tiles of 128 positions (64 for F16)
    ("F8", False, 16, 2, 512, [1, 128, 1029], 0, 0.0, 0),
    ("F8", True, 10, 1, 512, [300, 129], 0, 0.0, 2),
    ("F16", False, 16, 2, 512, [64, 65, 700], 100, 50.0, 0),
    ("F16", False, 2, 2, 512, [2000], 0, 0.0, 1),
    ("F8", False, 8, 8, 64, [1, 2500, 127], 0, 0.0, 0),
    ("F8", True, 24, 2, 64, [129, 31], 0, 30.0, 0),
])
def test_wide_shapes_match_the_cuda_core_kernel(ctx, dtype, scaled, hq, hkv, d, lens, window, softcap, n_splits):
    import torch
    n, longest, n_layers = len(lens), max(lens), 2
    rng = np.random.default_rng(longest)
    gen = torch.Generator(device="cuda").manual_seed(longest)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(n_layers, hkv, d, longest + 3, n_slots=n + 1, scale_mode=int(scaled)),
                       vf.KvDtype[dtype])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, max_batch=n, n_splits=n_splits)
    if window:
        fwd.sliding_layers, fwd.sliding_window = set(range(n_layers)), window
    fwd.softcap = softcap
    try:
        for layer in range(n_layers):
            for i, length in enumerate(lens):
                kv = to_dev(kv_values(rng, (2, length, hkv, d)))
                fwd.b_step_kv_write(layer, kv[0], kv[1], length, 0, i)
        q = torch.randn(n_layers, n, hq, d, device="cuda", generator=gen)
        k, v = (to_dev(kv_values(rng, (n_layers, n, hkv, d))) for _ in range(2))
        pos = to_dev(np.array([x - 1 for x in lens], np.uint32))
        want, step, token = (torch.zeros_like(q) for _ in range(3))
        ctx.set_attn_impl(1)
        for layer in range(n_layers):
            fwd.decode_step(layer, q[layer], k[layer], v[layer], want[layer], None, pos, n, longest)
        ctx.set_attn_impl(0)
        for layer in range(n_layers):
            fwd.decode_step(layer, q[layer], k[layer], v[layer], step[layer], None, pos, n, longest)
        fwd.decode_token(q, k, v, token, None, pos, n, longest)
        torch.cuda.synchronize()
        ctx.poll()
        scale = max(1.0, float(want.abs().max()))
        assert float((step - want).abs().max()) < 2e-5 * scale
        assert float((token - want).abs().max()) < 2e-5 * scale
    finally:
        ctx.set_attn_impl(0)
        fwd.workspace.destroy()
        cache.destroy()


def test_impl_3_decodes_as_0(ctx):
    """attn_impl 3 differs from 0 in prefill only: the same kernel, so the same bits (the CUDA-core kernel's are others)."""
    import torch
    hq, hkv, d, L = 16, 2, 512, 700
    gen = torch.Generator(device="cuda").manual_seed(3)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L), vf.KvDtype.F16)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    try:
        kv = torch.randn(2, L, hkv, d, device="cuda", generator=gen)
        fwd.b_step_kv_write(0, kv[0], kv[1], L, 0)
        q, got = torch.randn(hq, d, device="cuda", generator=gen), {}
        for impl in (0, 1, 3):
            ctx.set_attn_impl(impl)
            got[impl] = torch.zeros_like(q)
            fwd.step_attention(0, q, got[impl], L - 1)
        torch.cuda.synchronize()
        assert torch.equal(got[3], got[0]) and not torch.equal(got[1], got[0])
    finally:
        ctx.set_attn_impl(0)
        fwd.workspace.destroy()
        cache.destroy()
