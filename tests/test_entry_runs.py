"""Entry positions near the end of what an int can count (fiim_internal.h, EntryRun): a walk over a run of
entries ends, and tells every entry of its steps from the places past the end."""
import os
import subprocess

import pytest

from conftest import PKG, ROOT

PROGRAM = r"""
#include "fiim_internal.h"
#include <climits>
#include <cstdio>
int main() {
    const int ends[] = {0, 1, 31, 32, 33, 255, 256, 257, INT_MAX - 256, INT_MAX - 255, INT_MAX - 33, INT_MAX - 1, INT_MAX};
    const int lens[] = {0, 1, 31, 32, 33, 255, 256, 257, 1000};
    for (int step : {32, 256})
        for (int e : ends)
            for (int len : lens) {
                if (len > e) continue;
                const int b = e - len;
                long steps = 0, seen = 0;
                for (fiim::EntryRun t(b, e); t.more(); t.next(step)) {
                    const long at = b + steps * (long)step;
                    if ((long)t.at != at || ++steps > len) return 1;
                    for (int k = 0; k < step; ++k) {
                        if (t.has(k) != (at + k < (long)e)) return 2;
                        seen += t.has(k);
                    }
                }
                if (seen != len) return 4;
            }
    std::puts("ok");
    return 0;
}
"""


def test_runs_near_the_last_entry(tmp_path):
    if not os.path.exists("/usr/local/cuda/include/cuda_runtime.h"):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "runs.cpp", str(tmp_path / "runs")
    src.write_text(PROGRAM)
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover", f"-I{PKG}/csrc",
                    f"-I{ROOT}/include", "-I/usr/local/cuda/include", str(src), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout == "ok\n"
