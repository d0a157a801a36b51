"""The split count that the decode kernel chooses by itself, and the sequences that it gives to a warp each, asked of the library's
own functions: no GPU needed."""
import os
import shutil
import subprocess

import pytest

import vulkanforge_b200 as vf

CSRC = os.path.join(os.path.dirname(os.path.abspath(vf.__file__)), "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
DRIVER = r"""
#include <cstdio>
#include "common.cuh"
int main()
{
    vfkv_ctx ctx;
    ctx.sm_count = 148;
    unsigned dtype, hq, hkv, d, layers, seqs, hint;
    while (scanf("%u %u %u %u %u %u %u", &dtype, &hq, &hkv, &d, &layers, &seqs, &hint) == 7) {
        const uint32_t positions = 0;                      // the lengths are on the device: any address
        vfkv::AttnArgs a;
        a.kv.dtype = decltype(a.kv.dtype)(dtype); a.kv.n_kv_heads = hkv; a.kv.head_dim = d; a.kv.max_seq = hint;
        a.n_q_heads = hq; a.seq.n_seqs = seqs; a.seq.n_layers = layers; a.seq.positions = &positions; a.seq.max_len_hint = hint;
        printf("%u %u\n", vfkv::choose_splits(&ctx, a, 128), vfkv::one_warp_tiles(&ctx, dtype, d, uint64_t(layers) * seqs * hkv));
    }
}
"""


@pytest.fixture(scope="module")
def splits(tmp_path_factory):
    vf.load()
    where = tmp_path_factory.mktemp("split_count")
    (where / "main.cu").write_text(DRIVER)
    lib = os.path.dirname(CSRC)
    subprocess.run([NVCC, "-std=c++17", "-ccbin", "/usr/bin/g++", "-I", CSRC, str(where / "main.cu"), "-o", str(where / "main"),
                    "-L", lib, "-l:libvfkv.so", "-Xlinker", "-rpath=" + lib], check=True, capture_output=True, timeout=300)

    def ask(dtype, hq, hkv, d, layers, seqs, hint):
        line = "%d %d %d %d %d %d %d\n" % (int(vf.KvDtype[dtype]), hq, hkv, d, layers, seqs, hint)
        out = subprocess.run([str(where / "main")], input=line, capture_output=True, text=True, check=True, timeout=60).stdout
        return [int(x) for x in out.split()]
    return ask


@pytest.mark.parametrize("dtype,hq,hkv,d,layers,seqs,hint,least,most", [
    # one sequence, many layers: all units are as long as the hint says
    ("F8", 32, 8, 128, 16, 1, 2500, 1, 1),
    ("F8", 32, 8, 128, 36, 1, 8192, 1, 1),
    ("F16", 16, 8, 256, 16, 1, 2500, 2, 2),
    ("F8", 16, 8, 256, 2, 1, 9000, 18, 18),                # two more than the rules allow
    # several sequences: fewer splits than by the rules where that costs a long one among short ones little ...
    ("F8", 32, 8, 128, 4, 8, 4099, 1, 1),
    ("F16", 16, 8, 256, 4, 8, 1000, 1, 1),
    ("F8", 32, 8, 128, 2, 7, 3564, 1, 1),
    ("F8", 32, 8, 128, 1, 8, 9906, 2, 2),
    ("F8", 32, 8, 128, 1, 3, 9000, 6, 6),
    ("F8", 64, 8, 128, 5, 3, 5000, 1, 1),
    ("F16", 64, 8, 128, 5, 3, 5000, 1, 1),
    # ... and the rules' count where it would keep a few CTAs busy alone
    ("F8", 32, 8, 128, 4, 4, 16384, 8, 9),
    ("F8", 32, 8, 128, 1, 16, 16384, 8, 9),
    ("F8", 32, 8, 128, 4, 8, 8192, 8, 8),
    ("F8", 64, 8, 128, 4, 4, 16384, 8, 9),
    ("F16", 32, 8, 128, 2, 4, 20000, 8, 9),
    # more than two CTAs an SM without splits: none up to 8192 positions
    ("F8", 32, 8, 128, 10, 4, 4096, 1, 1),
])
def test_count(splits, dtype, hq, hkv, d, layers, seqs, hint, least, most):
    assert least <= splits(dtype, hq, hkv, d, layers, seqs, hint)[0] <= most


@pytest.mark.parametrize("dtype,d,pairs,tiles", [
    ("F8", 128, 444, 0), ("F8", 128, 445, 8), ("F8", 128, 888, 8), ("F8", 128, 889, 12), ("F8", 128, 1110, 12), ("F8", 128, 1111, 16),
    ("F16", 128, 444, 0), ("F16", 128, 445, 10), ("F16", 128, 888, 10), ("F16", 128, 889, 16), ("F16", 128, 65535, 16),
    ("F8", 256, 444, 0), ("F8", 256, 445, 8), ("F8", 256, 592, 8), ("F8", 256, 593, 12), ("F8", 256, 740, 12), ("F8", 256, 741, 16),
    ("F16", 256, 592, 8), ("F16", 256, 593, 16), ("F16", 64, 592, 0), ("F16", 64, 593, 8), ("F16", 64, 1184, 8), ("F16", 64, 1185, 12),
    ("F16", 64, 1480, 12), ("F16", 64, 1481, 16),
])
def test_tiles_of_a_sequence_for_a_warp(splits, dtype, d, pairs, tiles):
    assert splits(dtype, 1, 1, d, 1, pairs, 100)[1] == tiles
