"""vfkv_merge_partials at the edges of its groups of parts (four a warp, sixteen a round) and of dims (128 a block)."""
import pytest

import vulkanforge_b200 as vf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("n_parts,rows,d", [(0, 3, 128), (1, 3, 64), (3, 2, 100), (16, 5, 128), (17, 4, 129), (300, 2, 512)])
def test_merge_of_any_number_of_parts(ctx, n_parts, rows, d, packed):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n_parts)
    m, l = torch.randn(n_parts, rows, device="cuda", generator=gen) * 5, torch.rand(n_parts, rows, device="cuda", generator=gen) + 0.1
    o = torch.randn(n_parts, rows, d, device="cuda", generator=gen)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, 1, 64, 16), vf.KvDtype.F16)
    fwd = vf.CudaForward(ctx, cache, n_heads=1)
    try:
        out = torch.full((rows, d), 7.0, device="cuda")
        # at least a word behind each pointer, so that none is null
        pad = lambda t: torch.cat([t.reshape(-1), torch.full((4,), float("nan"), device="cuda")])
        if packed:
            blocks = pad(torch.cat([m, l, o.reshape(n_parts, rows * d)], 1) if n_parts else m)
            fwd.merge_partials_packed(blocks, n_parts, rows, d, out)
        else:
            mm, ll, oo = pad(m), pad(l), pad(o)
            fwd.merge_partials(mm, ll, oo, n_parts, rows, d, out)
        torch.cuda.synchronize()
        if n_parts == 0:
            assert not out.any()
            return
        w = torch.exp(m.double() - m.double().max(0).values)
        want = (w[:, :, None] * o.double()).sum(0) / (w * l.double()).sum(0)[:, None]
        assert float((out - want).abs().max()) < 1e-5 * max(1.0, float(want.abs().max()))
    finally:
        fwd.workspace.destroy()
        cache.destroy()
