"""How the tensor-core weight gradient splits a batch over blocks (host code of wgrad_mma.cuh): every run of 32
slices in one block, at most 640 points to an accumulator, and a grid within the limit of its x dimension for
batches beyond 65535 (chain, site) pairs."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bafqmc_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "wgrad_mma.cuh"
int main(int argc, char** argv) {
    for (int i = 1; i + 1 < argc; i += 2) {
        const bq::WgradSplit w = bq::wgrad_split(atoi(argv[i]), atoll(argv[i + 1]));
        printf("%lld %d %lld\n", w.items, w.per, w.chunks);
    }
}
"""
SHAPES = [(3, 1), (3, 2304), (31, 7), (32, 144), (33, 5), (160, 2304), (160, 7282 * 36), (319, 9), (320, 65536 * 2),
          (321, 65536), (352, 65536), (400, 1821 * 36), (639, 3), (640, 65536), (641, 1), (700, 6), (3200, 65536),
          (50, 456 * 144)]


def test_split_covers_the_batch_within_the_grid(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "w.cu", tmp_path / "w"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)],
                   check=True, timeout=300)
    out = subprocess.run([str(exe), *(str(v) for sh in SHAPES for v in sh)], check=True, timeout=60, capture_output=True,
                         text=True).stdout.split("\n")
    for (L, pairs), line in zip(SHAPES, out):
        items, per, chunks = map(int, line.split())
        runs = -(-L // 32)
        assert items == pairs * runs
        assert (chunks - 1) * per < items <= chunks * per
        assert 9 * chunks < 2 ** 31
        # points of the fullest block: `per` consecutive runs, each pair's last one short
        length = [min(32, L - 32 * r) for r in range(runs)]
        span = length * (per // runs + 2)
        assert max(sum(span[r:r + per]) for r in range(runs)) <= 640, (L, per)
