"""Memory that the library shares between calls, when the calls come on several streams."""
import numpy as np
import pytest

import vulkanforge_b200 as vf

pytestmark = pytest.mark.gpu


def _attention(q, k, v, first):
    """float64 attention of queries at positions first.. over k and v."""
    import torch
    m, hq, d = q.shape
    L, hkv = k.shape[:2]
    s = torch.einsum("mhgd,lhd->hgml", q.double().view(m, hkv, hq // hkv, d), k.double()) / d ** 0.5
    s = s.masked_fill(torch.arange(L, device="cuda") > first + torch.arange(m, device="cuda")[:, None], -float("inf"))
    return torch.einsum("hgml,lhd->mhgd", s.softmax(-1), v.double()).reshape(m, hq, d)


def test_new_memory_is_clear_before_its_first_use(ctx):
    """A workspace and a stream's scratch, made while the default stream is busy and used on another one at once."""
    import torch
    hq, hkv, d, L, m = 32, 8, 128, 16384, 256                    # pieces put together by the launch itself, by flags
    gen = torch.Generator(device="cuda").manual_seed(4)
    k, v = (torch.randn(L, hkv, d, device="cuda", generator=gen).half().float() for _ in range(2))
    q = torch.randn(m, hq, d, device="cuda", generator=gen)
    own = vf.Context(0)
    own.set_attn_tuning(8, 3)
    cache = vf.KvCache(own, vf.KvCacheConfig(1, hkv, d, L), vf.KvDtype.F16)
    stream = torch.cuda.Stream()
    fwd = None
    try:
        out, row = torch.zeros_like(q), torch.zeros(1, hq, d, device="cuda")
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000_000)                           # some 0.1 s on the default stream
        fwd = vf.CudaForward(own, cache, n_heads=hq)
        fwd.stream = stream.cuda_stream
        fwd.b_step_kv_write(0, k, v, L, 0)
        torch.cuda._sleep(200_000_000)
        fwd.run_flash_attn_batch(0, q, out, m, L - m, L, 0, 0)
        fwd.step_attention(0, q[-1:], row, L - 1)
        torch.cuda.synchronize()
        own.poll()
        want = _attention(q, k, v, L - m)
        assert float((out - want).norm() / want.norm()) < 2e-3
        assert float((row - want[-1:]).norm() / want[-1:].norm()) < 1e-5
    finally:
        if fwd:
            fwd.workspace.destroy()
        cache.destroy()
        own.destroy()


def test_decode_behind_a_raw_read_out_into_its_rows(ctx):
    """Mode-2 attention reads ahead of its predecessor, but not when that is a read-out that fills the rows it reads."""
    import torch
    hq, hkv, d, L = 32, 8, 128, 65536
    gen = torch.Generator(device="cuda").manual_seed(8)
    src = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L), vf.KvDtype.F8)
    dst = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L), vf.KvDtype.F16)
    fill, read = vf.CudaForward(ctx, src, n_heads=hq), vf.CudaForward(ctx, dst, n_heads=hq)
    try:
        k, v = (torch.randn(L, hkv, d, device="cuda", generator=gen).to(torch.float8_e4m3fn).float() for _ in range(2))
        q = torch.randn(1, hq, d, device="cuda", generator=gen)
        fill.b_step_kv_write(0, k, v, L, 0)
        want = _attention(q, k, v, L - 1)
        for mode in (0, 2, 2):
            ctx.set_dependent_launch(mode)
            dst.zero_fill()
            out = torch.zeros_like(q)
            torch.cuda.synchronize()
            fill.run_kv_fp8_to_f16(src.k_buffer, dst.k_buffer, L * hkv * d)
            fill.run_kv_fp8_to_f16(src.v_buffer, dst.v_buffer, L * hkv * d)
            read.step_attention(0, q, out, L - 1)
            torch.cuda.synchronize()
            assert float((out - want).norm() / want.norm()) < 2e-6
    finally:
        ctx.set_dependent_launch(0)
        for f, c in ((fill, src), (read, dst)):
            f.workspace.destroy()
            c.destroy()


def _short_prompt(ctx, n, seed):
    """A full-precision cache with 500 positions, n query chunks of 60 (two launches: tiles in shares, then the pieces)."""
    import torch
    hq, hkv, d, m, L = 32, 8, 128, 60, 500
    gen = torch.Generator(device="cuda").manual_seed(seed)
    cache = vf.KvCache(ctx, vf.KvCacheConfig(1, hkv, d, L), vf.KvDtype.F32)
    fwd = vf.CudaForward(ctx, cache, n_heads=hq)
    kv = torch.randn(2, L, hkv, d, device="cuda", generator=gen)
    fwd.b_step_kv_write(0, kv[0], kv[1], L, 0)
    qs = [torch.randn(m, hq, d, device="cuda", generator=gen) for _ in range(n)]
    want = [_attention(q, kv[0], kv[1], L - m) for q in qs]
    torch.cuda.synchronize()
    return cache, fwd, qs, want, lambda q, o: fwd.run_flash_attn_batch(0, q, o, m, L - m, L, 0, 0)


def test_every_stream_gets_scratch(ctx):
    """Streams that come and go, more than there are buffers: each call leaves its pieces and no two use one buffer at once."""
    import torch
    own = vf.Context(0)
    cache, fwd, qs, want, run = _short_prompt(own, 7, 5)
    try:
        for _ in range(3):
            got = [torch.zeros_like(q) for q in qs]
            streams = [torch.cuda.Stream() for _ in qs]
            for _ in range(4):
                for q, o, s in zip(qs, got, streams):
                    fwd.stream, before = s.cuda_stream, own.launch_count()
                    run(q, o)
                    assert own.launch_count() - before == 2
            torch.cuda.synchronize()
            assert all(float((a - b).abs().max()) < 1e-5 for a, b in zip(got, want))
    finally:
        fwd.stream = None
        fwd.workspace.destroy()
        cache.destroy()
        own.destroy()


def test_captured_calls_share_no_scratch(ctx):
    """Two recordings of a short prompt, replayed beside each other and beside a call that leaves pieces."""
    import torch
    cache, fwd, qs, want, run = _short_prompt(ctx, 3, 6)
    try:
        got = [torch.zeros_like(q) for q in qs]
        streams, graphs = [torch.cuda.Stream() for _ in qs], []
        fwd.stream = streams[0].cuda_stream
        run(qs[0], got[0])                                       # the context has scratch
        torch.cuda.synchronize()
        for q, o, s in zip(qs[1:], got[1:], streams[1:]):
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                fwd.stream, before = s.cuda_stream, ctx.launch_count()
                run(q, o)
                assert ctx.launch_count() - before == 1          # in one piece
            graphs.append(g)
        for o in got:
            o.zero_()
        torch.cuda.synchronize()
        for _ in range(20):
            for g, s in zip(graphs, streams[1:]):
                with torch.cuda.stream(s):
                    g.replay()
            fwd.stream = streams[0].cuda_stream
            run(qs[0], got[0])
        torch.cuda.synchronize()
        assert all(float((a - b).abs().max()) < 1e-5 for a, b in zip(got, want))
    finally:
        fwd.stream = None
        fwd.workspace.destroy()
        cache.destroy()
