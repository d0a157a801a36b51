"""The kernel that the prefill dispatch takes for few items of 128-dim rows against the mma.sync kernel and the oracle:
pieces of unequal size, every mask, and the soft-cap on either side of its polynomial's range."""
import numpy as np
import pytest

import oracle
import vulkanforge_b200 as vf
from util import encode_cache, kv_values, rel_err, to_dev

pytestmark = pytest.mark.gpu
ODT = {"F16": oracle.F16, "F8": oracle.F8}


@pytest.mark.parametrize("dtype,hq,hkv,m,q_start,kv_start,window,softcap,q_gain", [
    ("F8", 32, 8, 64, 1500, 0, 0, 0.0, 1.0),       # 8 items of 13 tiles
    ("F16", 32, 8, 333, 1000, 0, 0, 0.0, 1.0),     # 48 items of up to 11 tiles
    ("F8", 32, 8, 100, 3000, 0, 700, 0.0, 1.0),    # window
    ("F8", 64, 8, 40, 2000, 300, 0, 0.0, 1.0),     # kv_start; g = 8
    ("F16", 8, 1, 300, 600, 0, 0, 30.0, 1.0),      # one kv-head; early row blocks have fewer tiles
    ("F8", 32, 8, 64, 2500, 0, 0, 50.0, 12.0),     # scores beyond the cap
    ("F16", 32, 8, 70, 1300, 1310, 0, 0.0, 1.0),   # early queries see nothing -> zeros
])
def test_few_items_match_mma_sync_and_the_oracle(ctx, dtype, hq, hkv, m, q_start, kv_start, window, softcap, q_gain):
    import torch
    d, L = 128, q_start + m
    rng = np.random.default_rng(m + q_start)
    frac = 0.01 if dtype == "F8" else 0.0
    k, v = kv_values(rng, (L, hkv, d), frac), kv_values(rng, (L, hkv, d), frac)
    q = rng.standard_normal((m, hq, d), dtype=np.float32) * np.float32(q_gain)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L), vf.KvDtype[dtype])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, softcap=softcap)
    try:
        fwd.b_step_kv_write(0, to_dev(k), to_dev(v), L, 0)
        outs = {}
        for impl in (0, 3):
            ctx.set_attn_impl(impl)
            out = torch.full((m, hq, d), float("nan"), device="cuda")
            for _ in range(2):
                fwd.run_flash_attn_batch(0, to_dev(q), out, m, q_start, L, 0, kv_start, window=window)
            torch.cuda.synchronize()
            ctx.poll()
            outs[impl] = out.cpu().numpy()
        assert rel_err(outs[0], outs[3]) < 5e-3
        kc, vc = encode_cache(k, ODT[dtype]), encode_cache(v, ODT[dtype])
        for i in (0, 1, m // 2, m - 1):
            causal = q_start + i + 1
            lo = min(causal, max(kv_start, causal - window) if window and causal > window else kv_start)
            want = oracle.attention_ref(q[i], kc, vc, ODT[dtype], hq, hkv, d, causal, lo, None, softcap) if lo < causal \
                else np.zeros((hq, d), np.float32)
            assert float(np.max(np.abs(outs[0][i] - want))) < (3e-2 * max(float(np.max(np.abs(want))), 1e-3) if dtype == "F8" else 2e-3)
    finally:
        ctx.set_attn_impl(0)
        fwd.workspace.destroy()
        cache.destroy()
