"""The shared allocations of a handle's small arrays (mage_b200/csrc/gam_slab.h),
compiled for the host with an allocator that fails at a chosen call: a failure is
not lost when later arrays still fit the rest of an allocation, nothing is given out
after it, arrays are 512-byte aligned and do not overlap."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "gam_slab.h"
int main() {
    const size_t big = GamSlab::SLAB / 4;
    // as a handle asks for them: large ones, then one that needs a new slab, then tiny ones
    const size_t want[] = {100, big - 512, big - 512, big - 512, 5 * big, big - 512, 3 * big / 4, 128, 400, big, 24};
    const int n = sizeof(want) / sizeof(want[0]);
    int total = 0;
    for (int bad = -1; bad < 8; bad++) {  // the call that fails
        GamSlab s;
        int calls = 0, err = 0, first = n;
        char* base = (char*)(size_t)(1 << 20);  // addresses only: nothing is touched
        std::vector<char*> at, mem;
        std::vector<size_t> size;
        for (int q = 0; q < n; q++) {
            char* p = (char*)s.take(want[q], err, [&](void** r, size_t bytes) {
                if (calls++ == bad) return 2;
                *r = base;
                mem.push_back(base);
                size.push_back(bytes);
                base += bytes + 4096;
                return 0;
            });
            if (err && first == n) first = q;
            if ((p != nullptr) != (q < first)) return printf("array %d of fail %d\n", q, bad), 1;
            if (!p) continue;
            bool in = false;
            for (size_t m = 0; m < mem.size(); m++) in |= p >= mem[m] && p + want[q] <= mem[m] + size[m];
            for (size_t m = 0; m < at.size(); m++)
                if (p < at[m] + want[m] && at[m] < p + want[q]) return printf("overlap\n"), 1;
            if (!in || (size_t)p % 512) return printf("place\n"), 1;
            at.push_back(p);
        }
        if (bad >= 0 && bad < calls && !err) return printf("failure %d lost\n", bad), 1;
        if (bad < 0) total = calls;
    }
    printf("%d\n", total);
    return total >= 3 && total < n ? 0 : 1;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_a_failed_allocation_is_reported(tmp_path):
    src, exe = tmp_path / "s.cpp", tmp_path / "s"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "mage_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
