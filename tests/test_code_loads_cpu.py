"""Loads of 16-bit code rows (fzb_codeload.cuh) compiled for the host: no element
past the array is touched, at any place, count and alignment, and the packed
codes are the array's."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "fzb_codeload.cuh"
#include <algorithm>
#include <cstdio>
#include <vector>
struct Checked {
    const uint16_t* p;
    uint32_t n;
    mutable int* bad;
    uint32_t g;
    Checked from(uint32_t to) const { return {p, n, bad, to}; }
    uint32_t at(int i) const { if (g + i >= n) { ++*bad; return 0xdeadu; } return p[g + i]; }
    uint32_t u16(int i) const { return at(i); }
    uint32_t u32(int i) const { if ((g + i) & 1u) ++*bad; return at(i) | at(i + 1) << 16; }
    uint2 u64(int i) const { if ((g + i) & 3u) ++*bad; return {u32(i), u32(i + 2)}; }
    uint2 u64_once(int i) const { return u64(i); }
    uint4 u128_once(int i) const {
        if ((g + i) & 7u) ++*bad;
        const uint2 a = u64(i), b = u64(i + 4);
        return {a.x, a.y, b.x, b.y};
    }
    uint32_t shift(uint32_t lo, uint32_t hi, uint32_t bits) const {
        return (uint32_t)((((uint64_t)hi << 32) | lo) >> bits);
    }
};
int main() {
    int bad = 0, wrong = 0, seen = 0;
    for (uint32_t n = 1; n <= 41; n++) {
        std::vector<uint16_t> c(n);
        for (uint32_t i = 0; i < n; i++) c[i] = (uint16_t)(0x8001u + 257u * i);
        const Checked src{c.data(), n, &bad, 0};
        for (uint32_t g = 0; g < n; g++) {
            for (int valid = 0; valid <= (int)std::min(8u, n - g); valid++) {
                auto want = [&](int i) { return i < valid ? (uint32_t)c[g + i] : 0u; };
                const bool last = g + valid == n;  // the end of a field of n codes
                for (int mode = 0; mode < 4; mode++) {
                    if ((mode == 0 && (g % 8 || valid % 8)) || (mode == 1 && (g % 4 || valid % 4))) continue;
                    uint32_t w[4];
                    fzb::load8(src, g, valid, fzb::end_mode(mode, last, n), w);
                    for (int i = 0; i < 4; i++) wrong += w[i] != (want(2 * i) | want(2 * i + 1) << 16);
                    seen++;
                }
                for (int mode = 0; mode < 3 && valid <= 4; mode++) {
                    if (mode < 2 && (g % 4 || valid % 4)) continue;
                    const uint2 w = fzb::load4(src, g, valid, mode);
                    wrong += w.x != (want(0) | want(1) << 16) || w.y != (want(2) | want(3) << 16);
                    seen++;
                }
            }
        }
    }
    std::printf("%d %d %d\n", bad, wrong, seen);
    return 0;
}
"""


def test_no_code_past_the_array_is_read(tmp_path):
    src, exe = tmp_path / "loads.cpp", tmp_path / "loads"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-w", "-std=c++17", "-I", os.path.join(ROOT, "fzgpumodules_b200", "csrc"),
                    "-I", "/usr/local/cuda/include", "-o", str(exe), str(src)], check=True)
    bad, wrong, seen = map(int, subprocess.run([str(exe)], check=True, capture_output=True).stdout.split())
    assert seen > 10000 and bad == 0 and wrong == 0
