"""The float TBC's staged stretch of a line (csrc/tbc_stage.hpp), built as plain C++."""
import os
import subprocess

from conftest import PKG

# Every float that the kernel's copies and its lanes' loads touch, in 64-bit
# arithmetic, for lines in the middle, at both ends and outside of spans, and
# positions saturated at the ends of the int range; -ftrapv aborts on a sum that wraps.
SOURCE = r"""
#include <climits>
#include <cstdint>
#include <cstdio>
#include <vector>
#include "tbc_stage.hpp"
int main() {
    long staged = 0, plain = 0;
    for (int n : {1, 16, 25, 26, 40, 30720, 61440, 61443, 921600}) {
        std::vector<int> at{INT_MIN, INT_MIN + 7, -1000000, -1, 0, INT_MAX - 26, INT_MAX - 7, INT_MAX};
        for (int d = -40; d <= 40; d++)
            for (int base : {7, n / 2, n / 2 + 2500, 30720, n}) at.push_back(base + d);
        for (int cap : {60, 2700, 12288})
            for (int first : at)
                for (int last : at) {
                    const vhsd::TbcStretch s = vhsd::tbc_stretch(first, last, n, cap);
                    const int64_t low = first < last ? first : last, high = first < last ? last : first;
                    if (!s.staged) {
                        plain++;
                        // a line well inside the span and the stage is staged
                        if (low >= 7 && high <= n - 26 && high - low + 36 <= cap) return std::printf("left out %d %d %d %d\n", first, last, n, cap), 1;
                        continue;
                    }
                    staged++;
                    const int64_t lo = s.lo, len = s.len;
                    if (lo % 4 || len % 4 || lo < 0 || len <= 0 || lo + len > n || len + 4 > cap)
                        return std::printf("copy %d %d %d %d\n", first, last, n, cap), 1;
                    for (int offset = 0; offset < 4; offset++) {
                        const int64_t lo2 = lo - ((lo + offset) & 3);
                        if (lo2 + len + 4 > n) return std::printf("chroma copy %d %d %d %d\n", first, last, n, cap), 1;
                        for (int64_t x : {low, high}) {
                            const int64_t a = x - 7 - lo, a2 = x - 7 - lo2;   // five groups of four from there
                            if (a < 0 || (a & ~3) + 20 > len || a2 < 0 || (a2 & ~3) + 20 > len + 4)
                                return std::printf("taps %d %d %d %d\n", first, last, n, cap), 1;
                        }
                    }
                }
    }
    return staged > 1000 && plain > 1000 ? 0 : 2;
}
"""


def test_staged_stretch_lies_in_the_span(tmp_path):
    src, exe = tmp_path / "stage.cpp", tmp_path / "stage"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ftrapv", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
