"""The f32 tiles of chunked prefill (attn_prefill_f32.cu): every cache type at the edges of its tiles
(64 rows, 64 positions), its shares (a block's tiles cut over several CTAs, several blocks in one) and its masks."""
import numpy as np
import pytest

import oracle
import vulkanforge_b200 as vf
from util import dev_view_bytes, encode_cache, kv_values, to_dev

pytestmark = pytest.mark.gpu
ODT = {"F32": oracle.F32, "F16": oracle.F16, "F8": oracle.F8, "F8s": oracle.F32}


@pytest.mark.parametrize("dtype,hq,hkv,d,m,q_start,kv_start,window,softcap", [
    ("F32", 32, 8, 128, 1, 0, 0, 0, 0.0),          # one row block of four rows, one position
    ("F32", 32, 8, 128, 16, 47, 0, 0, 0.0),        # exactly one tile of rows and one of positions
    ("F32", 32, 8, 128, 17, 48, 0, 0, 0.0),        # one more of each
    ("F32", 8, 1, 128, 20, 900, 0, 0, 0.0),        # three blocks, a tile a CTA
    ("F32", 8, 8, 64, 70, 300, 0, 100, 30.0),      # g = 1, head_dim 64, window, soft-cap
    ("F32", 10, 2, 256, 33, 500, 7, 0, 0.0),       # g = 5 does not tile 64 rows
    ("F32", 16, 2, 512, 40, 130, 0, 0, 0.0),
    ("F32", 32, 8, 128, 80, 0, 50, 0, 0.0),        # early queries have an empty range -> zeros
    ("F16", 24, 8, 128, 50, 200, 0, 64, 0.0),
    ("F16", 16, 2, 512, 9, 70, 0, 0, 0.0),
    ("F8", 24, 8, 128, 50, 200, 0, 0, 50.0),
    ("F8s", 32, 8, 128, 100, 333, 0, 0, 0.0),      # a scale for each position and head
    ("F8s", 16, 8, 256, 30, 1000, 0, 256, 50.0),
    ("F8s", 64, 8, 128, 300, 700, 0, 0, 0.0),      # several blocks a CTA
])
def test_f32_tiles_match_the_oracle(ctx, dtype, hq, hkv, d, m, q_start, kv_start, window, softcap):
    import torch
    scaled, name = dtype == "F8s", dtype[:2] if dtype == "F8s" else dtype
    L = q_start + m
    rng = np.random.default_rng(L + d)
    frac = 0.01 if name == "F8" else 0.0
    k, v = kv_values(rng, (L, hkv, d), frac), kv_values(rng, (L, hkv, d), frac)
    q = rng.standard_normal((m, hq, d), dtype=np.float32)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(2, hkv, d, L + 5, n_slots=2, scale_mode=int(scaled)), vf.KvDtype[name])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, softcap=softcap)
    try:
        fwd.b_step_kv_write(1, to_dev(k), to_dev(v), L, 0, 1)
        out = torch.full((m, hq, d), 7.0, device="cuda")
        fwd.run_flash_attn_batch(1, to_dev(q), out, m, q_start, L, 1, kv_start, slot=1, window=window)
        torch.cuda.synchronize()
        if scaled:                                 # the reference reads the codes and scales that the append stored
            def rows(buf, scales):
                codes = dev_view_bytes(buf + cache.slot_offset_bytes(1, 1), L * hkv * d)
                at = (1 * 2 + 1) * (L + 5) * hkv * 4
                sc = dev_view_bytes(scales + at, L * hkv * 4).view(np.float32).reshape(L, hkv, 1)
                return oracle.kv_fp8_to_f16(codes).view(np.float16).astype(np.float32).reshape(L, hkv, d) * sc
            kc, vc = rows(cache.k_buffer, cache.k_scales), rows(cache.v_buffer, cache.v_scales)
        else:
            kc, vc = encode_cache(k, ODT[name]), encode_cache(v, ODT[name])
        want = oracle.batch_attention_ref(q, kc, vc, ODT[dtype], hq, hkv, d, m, q_start, L, kv_start, window,
                                          softcap=softcap)
        got = out.cpu().numpy()
        assert float(np.max(np.abs(got - want))) < 1e-5 * max(1.0, float(np.max(np.abs(want))))
    finally:
        fwd.workspace.destroy()
        cache.destroy()


def test_pieces_on_several_streams(ctx):
    """Calls that leave pieces may overlap on different streams of a context; a fifth stream takes over the
    scratch that was used longest ago."""
    import torch
    hq, hkv, d, m, L = 32, 8, 128, 60, 500
    gen = torch.Generator(device="cuda").manual_seed(1)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L), vf.KvDtype.F32)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    try:
        kv = torch.randn(2, L, hkv, d, device="cuda", generator=gen)
        fwd.b_step_kv_write(0, kv[0], kv[1], L, 0)
        qs = [torch.randn(m, hq, d, device="cuda", generator=gen) for _ in range(6)]
        want, got = ([torch.zeros_like(q) for q in qs] for _ in range(2))
        for q, o in zip(qs, want):
            fwd.run_flash_attn_batch(0, q, o, m, L - m, L, 0, 0)
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream() for _ in qs]
        for _ in range(3):
            for q, o, s in zip(qs, got, streams):
                fwd.stream = s.cuda_stream
                fwd.run_flash_attn_batch(0, q, o, m, L - m, L, 0, 0)
        torch.cuda.synchronize()
        assert all(float((a - b).abs().max()) < 1e-5 for a, b in zip(want, got))
    finally:
        fwd.stream = None
        fwd.workspace.destroy()
        cache.destroy()


@pytest.mark.parametrize("hq,hkv,d,m,L", [(32, 8, 128, 200, 700), (16, 8, 256, 60, 1500), (8, 8, 64, 200, 3000)])
def test_scores_of_a_hundred_keep_their_accuracy(ctx, hq, hkv, d, m, L):
    """A score of 100 in 32 bits is 4e-6 (half an ulp) off at best, and its p by as much; results average that over the
    positions and cancel what the p have in common.  Sums of sixteen products stay below 2^-19.5, one of all d does not."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(L)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L), vf.KvDtype.F32)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    try:
        k, v = (torch.randn(L, hkv, d, device="cuda", generator=gen) for _ in range(2))
        q = torch.randn(m, hq, d, device="cuda", generator=gen) * 25
        fwd.b_step_kv_write(0, k, v, L, 0)
        out = torch.zeros_like(q)
        fwd.run_flash_attn_batch(0, q, out, m, L - m, L, 0, 0)
        s = torch.einsum("mhgd,lhd->hgml", q.double().view(m, hkv, hq // hkv, d), k.double()) / d ** 0.5
        s = s.masked_fill(torch.arange(L, device="cuda") > L - m + torch.arange(m, device="cuda")[:, None], -float("inf"))
        want = torch.einsum("hgml,lhd->mhgd", s.softmax(-1), v.double()).reshape(m, hq, d)
        assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -19.5
    finally:
        fwd.workspace.destroy()
        cache.destroy()
