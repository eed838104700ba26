"""Maps larger than their links can name are refused before anything is
launched: build_ploc and build_lbvh on 2^27 + 1 leaves return
cudaErrorInvalidValue (on a machine without a GPU any call that got further
would return cudaErrorNoDevice or cudaErrorInsufficientDriver instead, and
with null buffers nothing could be written)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "upbp_ploc.cuh"
int main()
{
    using namespace upbp;
    BoxSource src{};
    BuildScratch sc{};
    PlocScratch ps{};
    ps.capacity = 0xffffffffu;
    ps.grid = 1;
    const unsigned* order = nullptr;
    unsigned launches = 0, outcome[kPcWords] = {};
    for (unsigned n : {kMaxBvhPrimitives + 1u, 0xfffffff0u}) {
        if (build_ploc(src, n, nullptr, sc, ps, nullptr, &order, &launches, outcome, kPlocPasses, 0) !=
            cudaErrorInvalidValue) return 1;
        if (build_lbvh(src, n, nullptr, sc, nullptr, &order) != cudaErrorInvalidValue) return 2;
    }
    return launches ? 3 : 0;
}
"""


def test_builds_refuse_more_leaves_than_links_hold(tmp_path):
    from gpuupbp_b200 import build
    src, exe = tmp_path / "limit.cu", tmp_path / "limit"
    src.write_text(PROGRAM)
    # -O0: host code alone is run
    subprocess.run([build.NVCC] + build.ARCH + ["-O0", "-std=c++17", "-ccbin", build.HOST_CXX, "-diag-suppress", "549,550",
                                                "-Xptxas", "-O0", "-I", build.CSRC, "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    # no device is visible to it, wherever the test runs
    assert subprocess.run([str(exe)], env=dict(os.environ, CUDA_VISIBLE_DEVICES="")).returncode == 0
