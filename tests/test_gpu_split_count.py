"""Tokens of nine to 295 (sequence, kv-head) pairs, whose split count the model of the launch finds (test_split_count_cpu.py has
the counts named here), against attention in 64 bits over the rows that the cache holds."""
import numpy as np
import pytest

import vulkanforge_b200 as vf
from util import dev_view_bytes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,scaled,hq,hkv,d,lens,n_layers,softcap", [
    ("F8", False, 32, 8, 128, [2500], 16, 0.0),                  # 128 pairs, one split
    ("F8", False, 64, 8, 128, [5000, 2531, 4001], 5, 30.0),      # one; heads on M; ragged last tiles and chains
    ("F8", True, 32, 8, 128, [4099, 2001, 3000, 2049], 8, 0.0),  # one
    ("F16", False, 16, 8, 256, [2500], 16, 50.0),                # two
    ("F16", False, 64, 8, 128, [5000, 129, 1], 5, 0.0),          # one, of very different lengths
    ("F8", False, 32, 8, 128, [9000, 700, 1], 1, 0.0),           # six, some of them empty
    ("F8", False, 16, 8, 256, [9000], 2, 0.0),                   # eighteen, more than the rules' sixteen
])
def test_counts_by_the_model_of_the_launch(ctx, dtype, scaled, hq, hkv, d, lens, n_layers, softcap):
    import torch
    n, longest = len(lens), max(lens)
    capacity = longest + 3
    gen = torch.Generator(device="cuda").manual_seed(longest)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(n_layers, hkv, d, capacity, n_slots=n, scale_mode=int(scaled)), vf.KvDtype[dtype])
    cache.zero_fill()
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, max_batch=n, softcap=softcap)
    try:
        for layer in range(n_layers):
            for i, length in enumerate(lens):
                kv = torch.randn(2, length, hkv, d, device="cuda", generator=gen)
                fwd.b_step_kv_write(layer, kv[0], kv[1], length, 0, i)
        q = torch.randn(n_layers, n, hq, d, device="cuda", generator=gen)
        k, v = (torch.randn(n_layers, n, hkv, d, device="cuda", generator=gen) for _ in range(2))
        pos = torch.tensor([x - 1 for x in lens], dtype=torch.int32, device="cuda")
        out = torch.zeros_like(q)
        fwd.decode_token(q, k, v, out, None, pos, n, longest)
        ctx.poll()
        torch.cuda.synchronize()

        def rows(buf, scales):
            raw = torch.from_numpy(dev_view_bytes(buf, cache.bytes_per_buffer())).cuda()
            x = raw.view(torch.float8_e4m3fn if dtype == "F8" else torch.float16).view(n_layers, n, capacity, hkv, d)
            if not scaled:
                return x, None
            s = dev_view_bytes(scales, n_layers * n * capacity * hkv * 4).view(np.float32).reshape(n_layers, n, capacity, hkv, 1)
            return x, torch.from_numpy(s.copy()).cuda().double()

        (kc, ks), (vc, vs) = rows(cache.k_buffer, cache.k_scales if scaled else 0), rows(cache.v_buffer, cache.v_scales if scaled else 0)
        wrong = all_of_it = 0.0
        for layer in range(n_layers):
            for i, length in enumerate(lens):
                kk, vv = kc[layer, i, :length].double(), vc[layer, i, :length].double()
                if scaled:
                    kk, vv = kk * ks[layer, i, :length], vv * vs[layer, i, :length]
                s = torch.einsum("hgd,phd->hgp", q[layer, i].double().view(hkv, hq // hkv, d), kk) / d ** 0.5
                if softcap:
                    s = softcap * torch.tanh(s / softcap)
                want = torch.einsum("hgp,phd->hgd", s.softmax(-1), vv).reshape(hq, d)
                wrong += float(((out[layer, i].double() - want) ** 2).sum())
                all_of_it += float((want ** 2).sum())
        # Q and P in two half-precision terms (2^-22 of a product each), sums in f32 over up to 9000 positions in chains: 3e-7 to 8e-7
        assert (wrong / all_of_it) ** 0.5 < 4e-6
    finally:
        fwd.workspace.destroy()
        cache.destroy()
