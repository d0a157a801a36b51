"""Chunked prefill over rows that are not finite: a query that sees such a row shows it, one that does not is as if the row
were not there -- also where both share a tile with it."""
import pytest

import vulkanforge_b200 as vf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,scaled,hq,hkv,d,m,q_start,window", [
    ("F8", True, 32, 8, 128, 100, 333, 0),          # one-tile kernel, whole
    ("F8", True, 32, 8, 128, 33, 5000, 0),          # in pieces
    ("F8", True, 24, 8, 64, 60, 700, 200),
    ("F8", False, 16, 8, 256, 100, 1100, 0),
    ("F16", False, 16, 8, 256, 150, 600, 300),
    ("F16", False, 8, 8, 64, 377, 708, 0),
    ("F32", False, 32, 8, 128, 60, 440, 100),       # f32 tiles
    ("F16", False, 16, 2, 512, 40, 130, 0),
])
def test_rows_that_are_not_finite(ctx, dtype, scaled, hq, hkv, d, m, q_start, window):
    import torch
    L = q_start + m
    gen = torch.Generator(device="cuda").manual_seed(L)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L, scale_mode=int(scaled)), vf.KvDtype[dtype])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    try:
        k, v = (torch.randn(L, hkv, d, device="cuda", generator=gen) for _ in range(2))
        if not scaled:
            to = {"F8": torch.float8_e4m3fn, "F16": torch.float16, "F32": torch.float32}[dtype]
            k, v = k.to(to).float(), v.to(to).float()
        nan = float("nan")
        v[L - m // 3, 1, 5] = nan                   # one element of V: that element of the outputs
        k[L - m // 5, 0, 3] = nan                   # one of K: all of them
        q = torch.randn(m, hq, d, device="cuda", generator=gen)
        fwd.b_step_kv_write(0, k, v, L, 0)
        if scaled:                                  # what the cache holds
            def stored(x):
                s = (x.nan_to_num(0.0).abs().amax(2, keepdim=True) * (1.0 / 448.0)).clamp_min(1e-12)
                return (x * (1.0 / s)).clamp(-448, 448).to(torch.float8_e4m3fn).float() * s
            k, v = stored(k), stored(v)
        out = torch.zeros_like(q)
        for _ in range(2):
            fwd.run_flash_attn_batch(0, q, out, m, q_start, L, 0, 0, window=window)
        g = hq // hkv
        for i in range(m):
            hi = q_start + i + 1
            lo = max(0, hi - window) if window else 0
            s = torch.einsum("hgd,lhd->hgl", q[i].double().view(hkv, g, d), k[lo:hi].double()) / d ** 0.5
            want = torch.einsum("hgl,lhd->hgd", s.softmax(-1), v[lo:hi].double()).reshape(hq, d)
            assert torch.equal(out[i].isnan(), want.isnan()), i
            fine = ~want.isnan()
            error = float((out[i].double() - want)[fine].abs().max())
            assert error < (1e-2 if dtype == "F8" and not scaled else 2e-3 if dtype == "F16" else 2e-5) * max(1.0, float(want[fine].abs().max())), i
    finally:
        fwd.workspace.destroy()
        cache.destroy()
