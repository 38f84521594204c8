"""Which NW batches run one warp per alignment (nw_run_warps), compiled for the
host: at each point both kernels were timed, and the rule has to take the one
that was faster by more than a fifth."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

# query length, band, alignments, the faster kernel
POINTS = [(150, 100, 256, "warp"), (150, 100, 4096, "warp"), (150, 70, 4096, "warp"), (150, 5, 512, "warp"),
          (150, 5, 2048, "thread"), (150, 5, 4096, "thread"), (150, 1, 1536, "thread"), (150, 20, 1536, "warp"),
          (150, 20, 4096, "thread"), (250, 100, 4096, "warp"), (250, 20, 1024, "warp"), (250, 20, 2560, "thread"),
          (250, 5, 1536, "thread"), (200, 50, 2048, "warp"), (200, 20, 4096, "thread"), (100, 100, 4096, "warp"),
          (100, 5, 1536, "warp"), (100, 5, 3584, "thread"), (36, 5, 2560, "thread"), (64, 30, 2560, "warp"),
          (75, 5, 512, "warp"), (75, 5, 3072, "thread"), (180, 20, 1536, "warp"), (180, 5, 4096, "thread")]

CHECK = r"""
#include "swb_internal.h"
#include <cstdio>
using namespace swb;
int main(int argc, char **argv) {
    const int cost = nw_i16_cost(1, 4, 6, 1, 6, 1);
    int q, w, n;
    while (std::scanf("%d %d %d", &q, &w, &n) == 3) {
        GlobalShape part[2], all;
        for (int k = 0; k < n; ++k) part[k & 1].add(q, q, w, cost);
        all.add(part[0]);
        all.add(part[1]);
        std::puts(nw_run_warps(all) ? "warp" : "thread");
    }
    // One wide alignment among many narrow ones: a thread's walk of it decides.
    GlobalShape mixed;
    for (int k = 0; k < 4000; ++k) mixed.add(150, 150, 5, cost);
    std::puts(nw_run_warps(mixed) ? "warp" : "thread");
    mixed.add(150, 150, 100, cost);
    std::puts(nw_run_warps(mixed) ? "warp" : "thread");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.exists("/usr/local/cuda/include/cuda_runtime.h"),
                    reason="needs g++ and the CUDA headers")
def test_rule_takes_the_faster_kernel(tmp_path):
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "swiftbwa_b200", "csrc"), "-I",
                    "/usr/local/cuda/include", "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], input="".join(f"{q} {w} {n}\n" for q, w, n, _ in POINTS), capture_output=True,
                       text=True, check=True)
    got = r.stdout.split()
    assert got == [p[3] for p in POINTS] + ["thread", "warp"], [(p, g) for p, g in zip(POINTS, got) if p[3] != g]
