"""Tokens of nine to 295 (sequence, kv-head) pairs, whose split count the model of the launch finds, against a decode step per
layer, whose counts come from the rules before it: other shapes, other chains of sums, the same products."""
import pytest

import vulkanforge_b200 as vf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,scaled,hq,hkv,d,lens,n_layers,softcap", [
    ("F8", False, 32, 8, 128, [2500], 16, 0.0),                  # 128 pairs
    ("F8", False, 64, 8, 128, [5000, 2531, 4001], 5, 30.0),      # heads on M; ragged last tiles and chains
    ("F8", True, 32, 8, 128, [4099, 2001, 3000, 2049], 8, 0.0),
    ("F16", False, 16, 8, 256, [2500], 16, 50.0),
    ("F16", False, 64, 8, 128, [5000, 129, 1], 5, 0.0),          # some of a sequence's splits are empty
])
def test_counts_by_the_model_of_the_launch(ctx, dtype, scaled, hq, hkv, d, lens, n_layers, softcap):
    import torch
    n, longest = len(lens), max(lens)
    gen = torch.Generator(device="cuda").manual_seed(longest)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(n_layers, hkv, d, longest + 3, n_slots=n, scale_mode=int(scaled)), vf.KvDtype[dtype])
    fwd = vf.CudaForward(ctx, cache, n_heads=hq, max_batch=n, softcap=softcap)
    try:
        for layer in range(n_layers):
            for i, length in enumerate(lens):
                kv = torch.randn(2, length, hkv, d, device="cuda", generator=gen)
                fwd.b_step_kv_write(layer, kv[0], kv[1], length, 0, i)
        q = torch.randn(n_layers, n, hq, d, device="cuda", generator=gen)
        k, v = (torch.randn(n_layers, n, hkv, d, device="cuda", generator=gen) for _ in range(2))
        pos = torch.tensor([x - 1 for x in lens], dtype=torch.int32, device="cuda")
        per_layer, together = torch.zeros_like(q), torch.zeros_like(q)
        for layer in range(n_layers):
            fwd.decode_step(layer, q[layer], k[layer], v[layer], per_layer[layer], None, pos, n, longest)
        fwd.decode_token(q, k, v, together, None, pos, n, longest)
        ctx.poll()
        torch.cuda.synchronize()
        # the same products, summed in f32 in other orders
        assert float((together - per_layer).abs().max()) <= 4e-6 * float(per_layer.abs().max())
    finally:
        fwd.workspace.destroy()
        cache.destroy()
