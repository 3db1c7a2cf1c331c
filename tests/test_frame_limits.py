"""The rule that admits a scene to the small-scene launches (frame_fits in
euc_kernels.cuh), compiled for the host: whatever it admits, the steps that
k_frame_raster counts and strides in 32 bits fit them with room for the grid's
warps.  No GPU is needed (nor used: a scene beyond the bound would keep one
busy for minutes)."""
import os
import shutil
import subprocess

import pytest

from euc_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include "euc_kernels.cuh"
using namespace eucg;
int main() {
    int bad = 0, taken = 0;
    const uint64_t max_warps = 1024ull * 64;  // more than any grid's
    auto check = [&](uint32_t n, uint32_t W, uint32_t H, uint32_t prim) {
        SceneDev s = {};
        s.ngroups = s.ntris = n;
        s.nverts = 3ull * std::min<uint32_t>(n, 40000);
        s.W = W;
        s.H = H;
        s.prim = prim;
        if (!frame_fits(s)) return;
        ++taken;
        // every primitive as many rows as the target has, or steps as its longer side
        const bool line = prim != EUC_PRIM_TRIANGLE_LIST;
        const uint64_t rows = line ? slot_items(s) : H, per = line ? 32 : 32 / kFrameLanes;
        uint64_t total = 0;
        for (uint64_t g = 0; g < n; g += 32)
            total += (std::min<uint64_t>(n - g, 32) * rows + per - 1) / per;
        if (total + max_warps > 0xFFFFFFFFull) {
            if (bad < 10) std::printf("%u primitives, %u x %u: %llu steps\n", n, W, H, (unsigned long long)total);
            ++bad;
        }
    };
    const uint32_t ns[] = {1, 31, 32, 33, 4096, 16384, 32767, 32768};
    for (uint32_t n : ns)
        for (uint32_t h : {1u, 2u, 480u, 1024u, 65534u, 65535u, 65536u, 1u << 18, 1u << 19, (1u << 20) - 1, 1u << 20})
            for (uint32_t w = 1; (uint64_t)w * h <= (1u << 20); w = w * 2 + 1)
                for (uint32_t prim : {(uint32_t)EUC_PRIM_TRIANGLE_LIST, (uint32_t)EUC_PRIM_LINE_LIST}) {
                    check(n, w, h, prim);
                    check(n, h, w, prim);
                }
    SceneDev s = {};
    s.ngroups = 32768;
    s.nverts = 98304;
    s.W = s.H = 1024;
    if (!frame_fits(s)) ++bad, std::printf("1024 x 1024 refused\n");
    std::printf("%d taken, %d over\n", taken, bad);
    return bad != 0 || taken == 0;
}
"""


def test_steps_of_every_admitted_scene_fit_32_bits(tmp_path):
    nvcc = build.nvcc()
    if not (os.path.exists(nvcc) or shutil.which(nvcc)):
        pytest.skip("nvcc not found")
    src = tmp_path / "limits.cu"
    src.write_text(SRC)
    exe = tmp_path / "limits"
    cmd = [nvcc] + build.ARCH + ["-O1", "-std=c++17", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"),
                                 "-I", os.path.join(ROOT, "euc_gb300", "csrc"), str(src), "-o", str(exe)]
    subprocess.run(cmd, check=True, capture_output=True, text=True, timeout=600)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout
