"""Which entry of the table of runs the aggregation's prep reads (pbe_internal.cuh:
window_first_entry): always one of its n + 1, whatever the two counters hold that the
pivots give (pivots that are no numbers give nothing). A host program; no GPU needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pbe-fixed-pivot-cuda_gb300", "csrc")

DRIVER = r"""
#include "pbe_internal.cuh"
#include <climits>
#include <cstdio>
using namespace pbe_gb300;
int main()
{
    const int odd[] = {INT_MIN, INT_MIN + 1, -1, 0, 1, 2, 3, 30, 63, 64, 65, 0x3fffffff, INT_MAX - 1, INT_MAX};
    for (int n : {1, 2, 3, 31, 64, 65, 500, 16384})
        for (int eh : odd)
            for (int el : odd) {
                const int e = window_first_entry(eh, el, n);
                const bool some = eh >= 1 && eh >= el;                  // descending runs eh .. max(el, 1)
                if (e != -1 && (e < 0 || e > n)) { std::printf("n=%d eh=%d el=%d: %d\n", n, eh, el, e); return 1; }
                if (some && eh < n && e != eh + 1) { std::printf("lost n=%d eh=%d el=%d\n", n, eh, el); return 1; }
                if (!some && e != -1) { std::printf("none n=%d eh=%d el=%d: %d\n", n, eh, el, e); return 1; }
            }
    // the table and the counters lie inside the scratch whose size callers are told
    for (int n : {1, 2, 31, 500, 3840}) {
        AggWs ws;
        char* base = reinterpret_cast<char*>(size_t(1) << 20);
        const size_t bytes = agg_ws_layout(n, base, &ws);
        if (bytes != agg_ws_bytes(n)) return 2;
        if (reinterpret_cast<char*>(ws.rend + n + 1) > base + bytes) return 3;
        if (reinterpret_cast<char*>(ws.counter + kAggCounters) > reinterpret_cast<char*>(ws.lpart)) return 4;
    }
    return 0;
}
"""


def test_window_entry_lies_in_the_table(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src, exe = tmp_path / "w.cu", tmp_path / "w"
    src.write_text(DRIVER)
    subprocess.run([nvcc, "-std=c++17", "-O1", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, (out.returncode, out.stdout)


def test_every_counter_is_cleared_before_the_tables():
    """counter[8], [9] and [10] are written by the pivots' threads alone."""
    with open(os.path.join(CSRC, "aggregation.cu")) as f:
        src = f.read()
    assert "cudaMemsetAsync(ws.counter, 0, kAggCounters * sizeof(int), s)" in src
