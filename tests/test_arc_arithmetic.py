"""Arc positions close to 2^31 (a graph may have up to 2^31 - 1 arcs): the number of segments of a row, the end of each and
the steps over it, computed by the library's own header compiled for the host. No GPU."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "show-me-dynamic-parallelism_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cstdint>
#include "dpg_kernels.h"
using namespace dpg;

// The segments of the row [b, e) cover it once, each of 1 to len arcs.
static int check(int64_t b, int64_t e, int len) {
    const int n = segments_of(static_cast<int>(e - b), len);
    if (n != (e - b + len - 1) / len) return 1;
    int64_t at = b;
    for (int k = n > 3 ? n - 3 : 0; k < n; ++k) {
        const int sb = static_cast<int>(b) + k * len;
        const int se = segment_end(sb, static_cast<int>(e), len);
        if (k > 0 && n > 3 && k == n - 3) at = sb;
        if (sb != at || se <= sb || se - sb > len) return 2;
        at = se;
    }
    return at == e ? 0 : 3;
}

int main() {
    const int64_t top = 2147483647;
    for (int len : {128, 256, 512})
        for (int64_t back = 0; back < 3 * len; ++back)
            for (int64_t e : {top, top - 1, top - len + 1, top - back})
                for (int64_t b : {int64_t{0}, e - back - 1, top - len - back}) {
                    if (b < 0 || b >= e) continue;
                    const int r = check(b, e, len);
                    if (r) {
                        std::printf("len %d row [%lld, %lld): %d\n", len, (long long)b, (long long)e, r);
                        return 1;
                    }
                }
    // A warp's rows, some of them hubs of a billion arcs: the rows kept are the longest prefix of at most 32 arcs.
    const int degs[] = {0, 1, 2, 5, 31, 32, 33, 1100000000, 2147483647};
    unsigned rnd = 1;
    for (int t = 0; t < 200000; ++t) {
        int incl = 0;
        int64_t sum = 0;
        for (int lane = 0; lane < 32; ++lane) {
            rnd = rnd * 1664525u + 1013904223u;
            const int d = degs[(rnd >> 16) % (t % 2 ? 9 : 4)];
            const int b = static_cast<int>(2147483647 - static_cast<int64_t>(d));
            incl = static_cast<int>(static_cast<unsigned>(incl) + static_cast<unsigned>(kept_degree(b, b + d)));
            sum += d;
            if ((incl <= 32) != (sum <= 32) || (sum <= 32 && incl != sum)) {
                std::printf("scan at lane %d: %d, %lld\n", lane, incl, (long long)sum);
                return 1;
            }
        }
    }
    return 0;
}
"""


def test_segments_near_2_31(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not shutil.which(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "arcs.cu", tmp_path / "arcs"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-O1", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I", str(CSRC), "-I",
                    str(ROOT / "include"), "-o", str(exe), str(src)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
