"""The tcgen05 prefill kernel with one Q tile of 128 rows a CTA: head_dim 64, 128 and 256, FP8 (plain and
with scales) and F16 rows, at the edges of its tiles (128 rows, 64 positions), cut into pieces and whole,
every mask, and the soft-cap on either side of its polynomial's range."""
import numpy as np
import pytest

import oracle
import vulkanforge_b200 as vf
from util import dev_view_bytes, encode_cache, kv_values, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,hq,hkv,d,m,q_start,kv_start,window,softcap,q_gain", [
    ("F16", 16, 8, 256, 64, 64, 0, 0, 0.0, 1.0),         # exactly one block of rows, two tiles
    ("F16", 16, 8, 256, 65, 130, 0, 0, 0.0, 1.0),        # one row block and one query
    ("F16", 16, 8, 256, 200, 1500, 0, 1024, 50.0, 1.0),  # window and soft-cap
    ("F16", 8, 8, 64, 300, 1000, 0, 0, 0.0, 1.0),
    ("F16", 8, 8, 64, 40, 3000, 17, 0, 30.0, 1.0),       # pieces; kv_start inside a tile
    ("F8", 16, 8, 256, 100, 2100, 0, 0, 0.0, 1.0),       # pieces
    ("F8", 16, 8, 256, 900, 100, 0, 0, 50.0, 20.0),      # scores beyond the cap; 120 blocks
    ("F8", 8, 8, 64, 130, 600, 0, 100, 0.0, 1.0),
    ("F8s", 32, 8, 128, 100, 333, 0, 0, 0.0, 1.0),
    ("F8s", 32, 8, 128, 33, 5000, 0, 0, 0.0, 30.0),      # pieces; peaked rows move the maximum and the scales' reference
    ("F8s", 16, 8, 256, 70, 900, 0, 256, 50.0, 1.0),
    ("F8s", 8, 8, 64, 200, 200, 0, 0, 0.0, 1.0),
    ("F8s", 24, 8, 128, 50, 1200, 0, 0, 0.0, 1.0),       # g = 3: a query's heads in two row blocks
    ("F8s", 64, 8, 128, 300, 700, 0, 0, 30.0, 1.0),
    ("F8s", 32, 8, 128, 80, 0, 50, 0, 0.0, 1.0),         # early queries have an empty range -> zeros
    ("F8s", 32, 8, 128, 1, 700, 0, 0, 0.0, 1.0),
])
def test_one_tile_kernel_matches_the_oracle(ctx, dtype, hq, hkv, d, m, q_start, kv_start, window, softcap, q_gain):
    import torch
    scaled, name = dtype == "F8s", dtype[:2] if dtype == "F8s" else dtype
    L = q_start + m
    rng = np.random.default_rng(L + d)
    frac = 0.01 if name == "F8" else 0.0
    k, v = kv_values(rng, (L, hkv, d), frac), kv_values(rng, (L, hkv, d), frac)
    if scaled:                                           # V scales that grow along the sequence by many binary orders
        v *= np.exp2(np.linspace(-6, 6, L, dtype=np.float32))[:, None, None]
    q = rng.standard_normal((m, hq, d), dtype=np.float32) * np.float32(q_gain)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(2, hkv, d, L + 5, n_slots=2, scale_mode=int(scaled)), vf.KvDtype[name])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, softcap=softcap)
    try:
        fwd.b_step_kv_write(1, to_dev(k), to_dev(v), L, 0, 1)
        out = torch.full((m, hq, d), float("nan"), device="cuda")
        for _ in range(2):
            fwd.run_flash_attn_batch(1, to_dev(q), out, m, q_start, L, 1, kv_start, slot=1, window=window)
        torch.cuda.synchronize()
        ctx.poll()
        if scaled:                                       # the reference reads the codes and scales that the append stored
            def rows(buf, scales):
                codes = dev_view_bytes(buf + cache.slot_offset_bytes(1, 1), L * hkv * d)
                sc = dev_view_bytes(scales + 3 * (L + 5) * hkv * 4, L * hkv * 4).view(np.float32).reshape(L, hkv, 1)
                return oracle.kv_fp8_to_f16(codes).view(np.float16).astype(np.float32).reshape(L, hkv, d) * sc
            odt, kc, vc = oracle.F32, rows(cache.k_buffer, cache.k_scales), rows(cache.v_buffer, cache.v_scales)
        else:
            odt = oracle.F16 if name == "F16" else oracle.F8
            kc, vc = encode_cache(k, odt), encode_cache(v, odt)
        got = out.cpu().numpy()
        assert np.isfinite(got).all()
        for i in sorted({0, 1, m // 3, m // 2, max(m - 2, 0), m - 1} & set(range(m))):
            causal = q_start + i + 1
            lo = min(causal, max(kv_start, causal - window) if window and causal > window else kv_start)
            want = oracle.attention_ref(q[i], kc, vc, odt, hq, hkv, d, causal, lo, None, softcap) if lo < causal \
                else np.zeros((hq, d), np.float32)
            top = max(1.0 if scaled else 1e-3, float(np.max(np.abs(want))))
            assert float(np.max(np.abs(got[i] - want))) < (1e-5 * top if scaled else 5e-3 * top if name == "F8" else 1e-3)
    finally:
        fwd.workspace.destroy()
        cache.destroy()


@pytest.mark.parametrize("hq,hkv,d,L", [(16, 8, 256, 200), (8, 8, 64, 1500)])
def test_rows_that_one_position_dominates(ctx, hq, hkv, d, L):
    """Position 100 outweighs position 10 by less than the kernel moves a row's maximum for, and all others by far: its
    p is not 1 but a number that half precision rounds by up to 2^-12, which the row's sum has to follow."""
    import torch
    m = 34
    rng = np.random.default_rng(d)
    k = np.zeros((L, hkv, d), np.float32)
    k[10, :, 0], k[100, :, 0] = 10.0, 11.0
    v = rng.standard_normal((L, hkv, d), dtype=np.float32).astype(np.float16).astype(np.float32)
    q = np.zeros((m, hq, d), np.float32)
    q[:, :, 0] = ((4.0 + 0.03 * np.arange(m)) * np.sqrt(d))[:, None]           # scores 40 .. 50 and a tenth more
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L), vf.KvDtype.F16)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    try:
        fwd.b_step_kv_write(0, to_dev(k), to_dev(v), L, 0)
        out = torch.zeros(m, hq, d, device="cuda")
        fwd.run_flash_attn_batch(0, to_dev(q), out, m, L - m, L, 0, 0)
        torch.cuda.synchronize()
        s = (q[:, 0, 0].astype(np.float64) / np.sqrt(np.float64(d)))[:, None] * k[:, 0, 0].astype(np.float64)      # [m][L]
        s[np.arange(L)[None] > (L - m + np.arange(m))[:, None]] = -np.inf
        p = np.exp(s - s.max(1, keepdims=True))
        p /= p.sum(1, keepdims=True)
        want = np.repeat(np.einsum("ml,lhd->mhd", p, v.astype(np.float64)), hq // hkv, axis=1)
        # the dominating p off by 2^-12 shifts the mean of the two rows by that share of the other's weight (at most e^-4)
        tol = 2.0 ** -12 * np.exp(-4.0) * np.abs(v[100] - v[10]).max() + 4e-6 * np.abs(v).max()
        assert np.abs(out.cpu().numpy() - want).max() < tol
    finally:
        fwd.workspace.destroy()
        cache.destroy()


@pytest.mark.parametrize("hq,hkv,m,q_start,softcap", [(64, 8, 166, 99, 0.0), (32, 8, 17, 485, 50.0), (32, 8, 60, 1000, 0.0)])
def test_short_f16_calls_take_q_in_two_terms(ctx, hq, hkv, m, q_start, softcap):
    """Q of one half-precision term moves a score s by up to 2^-12 |s| and each p by as much again; with two terms what is
    left is the rounding of p to half precision.  Queries 25 times larger (scores of some 70): 1e-3 or 5e-5."""
    import torch
    d, L = 128, q_start + m
    gen = torch.Generator(device="cuda").manual_seed(L)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L), vf.KvDtype.F16)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, softcap=softcap)
    try:
        k, v = (torch.randn(L, hkv, d, device="cuda", generator=gen).half().float() for _ in range(2))
        q = torch.randn(m, hq, d, device="cuda", generator=gen) * 25
        fwd.b_step_kv_write(0, k, v, L, 0)
        out = torch.zeros(m, hq, d, device="cuda")
        fwd.run_flash_attn_batch(0, q, out, m, q_start, L, 0, 0)
        s = torch.einsum("mhgd,lhd->hgml", q.double().view(m, hkv, hq // hkv, d), k.double()) / d ** 0.5
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(torch.arange(L, device="cuda") > q_start + torch.arange(m, device="cuda")[:, None], -float("inf"))
        want = torch.einsum("hgml,lhd->mhgd", s.softmax(-1), v.double()).reshape(m, hq, d)
        error = float((out.double() - want).norm() / want.norm())
        assert error < 2.0 ** -12                              # half an ulp of p at most, in the mean less
    finally:
        fwd.workspace.destroy()
        cache.destroy()


def test_more_row_blocks_than_a_grid_axis_holds(ctx):
    """65 541 blocks of 128 rows (one kv-head, 64 q-heads of 64): every query sees a window of 1024."""
    import torch
    hq, hkv, d, m = 64, 1, 64, 131080
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, m), vf.KvDtype.F8)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    try:
        gen = torch.Generator(device="cuda").manual_seed(2)
        k, v = (torch.randn(m, hkv, d, device="cuda", generator=gen).to(torch.float8_e4m3fn).float() for _ in range(2))
        fwd.b_step_kv_write(0, k, v, m, 0)
        q = torch.randn(m, hq, d, device="cuda", generator=gen)
        out = torch.full((m, hq, d), 7.0, device="cuda")
        fwd.run_flash_attn_batch(0, q, out, m, 0, m, 0, 0, window=1024)      # long enough a window for this kernel
        for i in (0, 1, 127, 70000, 131070, m - 1):
            lo = max(0, i + 1 - 1024)
            s = q[i].double() @ k[lo:i + 1, 0].double().T / d ** 0.5
            want = s.softmax(-1) @ v[lo:i + 1, 0].double()
            assert float((out[i] - want).norm() / want.norm()) < 5e-3
        assert bool(torch.isfinite(out).all()) and not bool((out == 7.0).all(2).any())
    finally:
        fwd.workspace.destroy()
        cache.destroy()


@pytest.mark.parametrize("dtype,hq,hkv,d,tiles", [(dt, hq, hkv, d, n) for dt, hq, hkv, d in
                                                  (("F8s", 32, 8, 128), ("F16", 16, 8, 256), ("F8", 16, 8, 256), ("F16", 8, 8, 64))
                                                  for n in ((1, 2, 3) if dt == "F8s" else (3,)) + (4, 5, 6, 9, 10)])
def test_a_reference_that_moves_in_every_tile(ctx, dtype, hq, hkv, d, tiles):
    """Scores that rise by 20 (29 binary orders) a tile of 64 positions for one query in three, fall for the next and stay for
    the third: the two groups of softmax warps, which take the even and the odd tiles, hand the reference maximum to and fro
    at every number of tiles around that of the score buffers (two and four).  P is rounded to half precision, its sum
    too (scales: neither), which moves a weighted mean of V by at most 2^-11 of the largest V on either side."""
    import torch
    scaled, name = dtype == "F8s", "F16" if dtype == "F16" else "F8"
    m, L = 35, tiles * 64 - 5
    rng = np.random.default_rng(tiles * d)
    k = np.zeros((L, hkv, d), np.float32)
    k[:, :, 0] = (np.arange(L) // 16)[:, None] * 0.25                          # exact in E4M3 up to 4, in F16 throughout
    if name == "F8":
        k[:, :, 0] = torch.from_numpy(k[:, :, 0].copy()).to(torch.float8_e4m3fn).float().numpy()
    v = torch.from_numpy(rng.standard_normal((L, hkv, d), dtype=np.float32)).to(torch.float8_e4m3fn).float().numpy()
    if scaled:                                                                  # scales are a power of two: nothing is rounded
        k[:, :, 1], v[:, :, 0] = 7.0, 448.0
        k *= 64.0
    slope = np.array([20.0, -20.0, 0.0], np.float32)[np.arange(m) % 3] * np.sqrt(np.float32(d)) / (64.0 if scaled else 1.0)
    q = np.zeros((m, hq, d), np.float32)
    q[:, :, 0] = slope[:, None]
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L, scale_mode=int(scaled)), vf.KvDtype[name])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    try:
        fwd.b_step_kv_write(0, to_dev(k), to_dev(v), L, 0)
        out = torch.full((m, hq, d), float("nan"), device="cuda")
        fwd.run_flash_attn_batch(0, to_dev(q), out, m, L - m, L, 0, 0)
        torch.cuda.synchronize()
        ctx.poll()
        s = (q[:, 0, 0].astype(np.float64) / np.sqrt(np.float64(d)))[:, None] * k[:, 0, 0].astype(np.float64)      # [m][L]
        s[np.arange(L)[None] > (L - m + np.arange(m))[:, None]] = -np.inf
        p = np.exp(s - s.max(1, keepdims=True))
        p /= p.sum(1, keepdims=True)
        want = np.repeat(np.einsum("ml,lhd->mhd", p, v.astype(np.float64)), hq // hkv, axis=1)
        top = np.abs(v).max(axis=(0, 1))
        tol = (2e-5 if scaled else 2.0 ** -10) * top + (1e-5 if scaled else 0.0)
        assert (np.abs(out.cpu().numpy() - want) <= tol).all()
    finally:
        fwd.workspace.destroy()
        cache.destroy()


@pytest.mark.parametrize("dtype,hq,hkv,d,lens", [("F16", 8, 8, 64, 1500), ("F16", 32, 8, 128, 700), ("F16", 16, 8, 256, 300), ("F8s", 32, 8, 128, 200),
                                                 ("F8s", 16, 8, 256, 130)])
def test_scores_beyond_what_f32_counts_in_units(ctx, dtype, hq, hkv, d, lens):
    """Scores of 2^8 to 2^31, most of them below zero, one position's far above the others': its row of V, whatever a unit in the
    maximum's last place is (2 from 2^24 on; half precision has nothing below 2^-24).  Only the calls whose Q is in two terms,
    scaled, hold such queries."""
    import torch
    scaled, name = dtype == "F8s", "F16" if dtype == "F16" else "F8"
    m = 48
    L = lens + m
    rng = np.random.default_rng(d + lens)
    k = np.zeros((L, hkv, d), np.float32)
    k[:, :, 0] = 128.0                                     # with q[0]: where all scores lie
    pick = lens // 2
    k[pick, :, 2] = 64.0
    v = torch.from_numpy(rng.standard_normal((L, hkv, d), dtype=np.float32)).to(torch.float8_e4m3fn).float().numpy()
    if scaled:
        v[:, :, 0] = 448.0                                 # scales of V are 1
        k *= 3.5                                           # of K too: 448 in every row
    q = np.zeros((m, hq, d), np.float32)
    size = np.exp2(np.linspace(8, 31, m))[:, None] * np.sqrt(d) * (1.0 + 0.4 * rng.random((m, hq)))
    sign = np.where(np.arange(m) % 5 == 4, 1.0, -1.0)[:, None]
    q[:, :, 0] = size * sign / k[0, 0, 0]
    q[:, :, 2] = size / 4 / 64.0
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L, scale_mode=int(scaled)), vf.KvDtype[name])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    try:
        fwd.b_step_kv_write(0, to_dev(k), to_dev(v), L, 0)
        out = torch.full((m, hq, d), float("nan"), device="cuda")
        fwd.run_flash_attn_batch(0, to_dev(q), out, m, lens, L, 0, 0)
        torch.cuda.synchronize()
        ctx.poll()
        want = np.broadcast_to(np.repeat(v[pick], hq // hkv, axis=0), (m, hq, d))
        # the other positions are e^-64 and further below
        assert float(np.abs(out.cpu().numpy() - want).max()) <= 1e-5 * float(np.abs(v).max())
    finally:
        fwd.workspace.destroy()
        cache.destroy()


@pytest.mark.parametrize("hq,hkv,d,L,gain", [(32, 8, 128, 300, 1.0), (32, 8, 128, 4000, 3.0), (16, 8, 256, 500, 2.0), (8, 8, 64, 300, 1.0)])
def test_v_scales_far_apart(ctx, hq, hkv, d, L, gain):
    """Eight positions whose V is 2^12 larger than the others' and whose p is e^-14 of theirs.  P times its V scale is fed as two
    half-precision terms, 2^-22 of it or the last bit of the second, which is 2^-34 of (the row's largest p x the largest V scale)."""
    import torch
    m = 35
    gen = torch.Generator(device="cuda").manual_seed(L)
    k, v = (torch.randn(L, hkv, d, device="cuda", generator=gen) for _ in range(2))
    k[:, :, 0] = 14.0
    sinks = torch.arange(8, device="cuda") * (L // 9) + 3
    k[sinks, :, 0] = 0.0
    v[sinks] *= 4096.0
    q = torch.randn(m, hq, d, device="cuda", generator=gen) * gain
    q[:, :, 0] = d ** 0.5
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L, scale_mode=1), vf.KvDtype.F8)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    try:
        fwd.b_step_kv_write(0, k, v, L, 0)
        out = torch.zeros(m, hq, d, device="cuda")
        fwd.run_flash_attn_batch(0, q, out, m, L - m, L, 0, 0)
        torch.cuda.synchronize()
        ctx.poll()

        def rows(buf, scales):                             # the codes and scales that the append stored
            codes = torch.from_numpy(dev_view_bytes(buf, L * hkv * d)).view(torch.float8_e4m3fn).view(L, hkv, d).cuda().double()
            return codes, torch.from_numpy(dev_view_bytes(scales, L * hkv * 4).view(np.float32).copy()).view(L, hkv, 1).cuda().double()

        (kc, ks), (vc, vs) = rows(cache.k_buffer, cache.k_scales), rows(cache.v_buffer, cache.v_scales)
        s = torch.einsum("mhgd,lhd->hgml", q.double().view(m, hkv, hq // hkv, d), kc * ks) / d ** 0.5
        s = s.masked_fill(torch.arange(L, device="cuda") > L - m + torch.arange(m, device="cuda")[:, None], -float("inf"))
        p = torch.exp(s - s.amax(-1, keepdim=True))
        total = p.sum(-1)[..., None]
        mean = lambda x: (torch.einsum("hgml,lhd->hgmd", p, x) / total).permute(2, 0, 1, 3).reshape(m, hq, d)
        want = mean(vc * vs)
        # two terms of every product, and 4e-6 of the sum for scores and exponentials in f32 (scores up to some 20)
        fed = torch.einsum("hgml,lhd->hgmd", (s > -1e30).double(), vc.abs()) * 2.0 ** -35 * vs.max() / total
        tol = fed.permute(2, 0, 1, 3).reshape(m, hq, d) + (2.0 ** -22 + 4e-6) * mean((vc * vs).abs())
        worst = float(((out.double() - want).abs() / tol).max())
        error = float((out.double() - want).norm() / want.norm())
        print("V scales far apart: %.2e of 64 bits, %.2f of the bound" % (error, worst))
        assert worst <= 1.0
    finally:
        fwd.workspace.destroy()
        cache.destroy()
