"""Tokens of many short sequences: a warp each, without splits or a merge, against a decode step per layer (whose grids are
small enough for CTAs of several warps), at the edges of the kernel's tiles and at the most tiles that this is done for
(test_split_count_cpu.py has the lines)."""
import numpy as np
import pytest

import vulkanforge_b200 as vf
from util import kv_values, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,scaled,hq,hkv,d,lens,window,softcap", [
    ("F8", False, 32, 8, 128, [1, 2, 31, 32, 33, 64, 65, 96], 0, 0.0),
    ("F8", False, 32, 8, 128, [512, 511, 1, 481, 480, 256, 300, 33], 0, 0.0),     # sixteen tiles of 32, three stages
    ("F8", False, 64, 8, 128, [64, 100, 7, 32, 161, 128, 127, 129], 0, 30.0),     # eight q-heads a kv-head: heads on M
    ("F8", True, 32, 8, 128, [70, 32, 1, 97, 128, 40, 64, 3], 0, 0.0),
    ("F8", False, 16, 8, 256, [1, 400, 33, 65, 32, 31, 500, 90], 100, 50.0),      # a window shorter than some
    ("F8", False, 32, 2, 128, [60] * 30 + [64, 1], 0, 0.0),                       # groups of sixteen, cut into parts
    ("F16", False, 32, 8, 128, [16, 17, 15, 1, 256, 240, 241, 33], 0, 0.0),
    ("F16", False, 16, 8, 256, [5, 16, 32, 33, 128, 200, 256, 1], 0, 50.0),
    ("F16", False, 8, 8, 64, [40, 1, 16, 17, 250, 31, 32, 64], 0, 0.0),
    ("F16", False, 16, 1, 128, [30] * 63 + [1], 0, 0.0),                          # sixteen q-heads in two rows of eight
])
def test_a_warp_a_sequence(ctx, dtype, scaled, hq, hkv, d, lens, window, softcap):
    import torch
    n, longest = len(lens), max(lens)
    n_layers = -(-1500 // (n * hkv))                       # above ten CTAs an SM: up to sixteen tiles
    rng = np.random.default_rng(longest + d)
    gen = torch.Generator(device="cuda").manual_seed(longest)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(n_layers, hkv, d, longest + 3, n_slots=n, scale_mode=int(scaled)), vf.KvDtype[dtype])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, max_batch=n, softcap=softcap, sliding_window=window,
                         sliding_layers=range(n_layers) if window else ())
    try:
        for layer in range(n_layers):
            for i, length in enumerate(lens):
                kv = torch.randn(2, length, hkv, d, device="cuda", generator=gen)
                fwd.b_step_kv_write(layer, kv[0], kv[1], length, 0, i)
        q = torch.randn(n_layers, n, hq, d, device="cuda", generator=gen)
        k, v = (to_dev(kv_values(rng, (n_layers, n, hkv, d))) for _ in range(2))
        pos = to_dev(np.array([x - 1 for x in lens], np.uint32))
        row = cache.row_bytes(0)

        def state():
            torch.cuda.synchronize()
            out = np.empty((2, cache.bytes_per_buffer()), np.uint8)
            for o, a in zip(out, (cache.k_buffer, cache.v_buffer)):
                ctx.check(ctx._lib.vfkv_memcpy_d2h(ctx.handle, o.ctypes.data, a, o.nbytes, None))
            ctx.check(ctx._lib.vfkv_stream_synchronize(ctx.handle, None))
            return [out[:, cache.slot_offset_bytes(l, s) + (x - 1) * row:][:, :row].copy()
                    for l in range(n_layers) for s, x in enumerate(lens)]

        per_layer, together = torch.zeros_like(q), torch.zeros_like(q)
        for layer in range(n_layers):
            fwd.decode_step(layer, q[layer], k[layer], v[layer], per_layer[layer], None, pos, n, longest)
        want = state()
        for layer in range(n_layers):                      # other rows in the token's place, to be overwritten again
            for i, length in enumerate(lens):
                z = torch.zeros(2, 1, hkv, d, device="cuda")
                fwd.b_step_kv_write(layer, z[0], z[1], 1, length - 1, i)
        fwd.decode_token(q, k, v, together, None, pos, n, longest)
        got = state()
        ctx.poll()
        assert all((a == b).all() for a, b in zip(got, want))
        # both sum the same products in f32, in other orders; sixteen heads of F16: P in one half-precision term, 2^-12 of it
        tol = (2.0 ** -11 if hq // hkv > 8 and dtype == "F16" else 4e-6) * float(per_layer.abs().max())
        assert float((together - per_layer).abs().max()) <= tol
    finally:
        fwd.workspace.destroy()
        cache.destroy()


@pytest.mark.parametrize("hq,hkv,d,lens", [(16, 1, 128, [30] * 63 + [1]), (24, 2, 256, [1, 16, 33, 100] * 8), (32, 2, 64, [17, 128, 250, 5] * 8)])
def test_groups_of_nine_to_sixteen_feed_p_in_two_terms(ctx, hq, hkv, d, lens):
    """Against attention in 64 bits of the Q that half precision holds: what is left is sums in f32 (P rounded to half precision as
    well: 1.5e-4)."""
    import torch
    n, longest = len(lens), max(lens)
    n_layers = -(-1500 // (n * hkv))                       # above ten CTAs an SM: up to sixteen tiles
    gen = torch.Generator(device="cuda").manual_seed(d)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(n_layers, hkv, d, longest, n_slots=n), vf.KvDtype.F16)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, max_batch=n)
    try:
        k, v = (torch.randn(n_layers, n, longest, hkv, d, device="cuda", generator=gen).half().float() for _ in range(2))
        for layer in range(n_layers):
            for i, length in enumerate(lens):
                fwd.b_step_kv_write(layer, k[layer, i, :length].contiguous(), v[layer, i, :length].contiguous(), length, 0, i)
        at = torch.tensor([x - 1 for x in lens], device="cuda")
        new_k, new_v = (torch.stack([x[:, i, length - 1] for i, length in enumerate(lens)], 1).contiguous() for x in (k, v))
        q = torch.randn(n_layers, n, hq, d, device="cuda", generator=gen)
        out = torch.zeros_like(q)
        fwd.decode_token(q, new_k, new_v, out, None, at.int(), n, longest)
        torch.cuda.synchronize()
        s = torch.einsum("lnhgd,lnphd->lnhgp", q.half().double().view(n_layers, n, hkv, hq // hkv, d), k.double()) / d ** 0.5
        s = s.masked_fill(torch.arange(longest, device="cuda") > at.view(1, n, 1, 1, 1), -float("inf"))
        want = torch.einsum("lnhgp,lnphd->lnhgd", s.softmax(-1), v.double()).reshape(out.shape)
        assert float((out.double() - want).norm() / want.norm()) < 4e-6
    finally:
        fwd.workspace.destroy()
        cache.destroy()
