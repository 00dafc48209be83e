"""Room for a frame graph's bin references (csrc/graph_bins.h), compiled here for the
host: every job whose frame fits 32-bit places gets at least that frame and half as
much again or four a tile, also where the usual 18 for one would pass 2^32, and only
larger ones are refused."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tg_gb300" / "csrc"
MAIN = r"""
#include "graph_bins.h"
#include <cstdio>
#include <cstdlib>
int main(int n, char** a)
{
    for (int i = 1; i + 1 < n; i += 2) {
        uint64_t c = 0;
        const bool ok = graph_bin_capacity(strtoull(a[i], 0, 10), strtoull(a[i + 1], 0, 10), &c);
        printf("%d %llu\n", (int)ok, (unsigned long long)c);
    }
}
"""
M = 2 ** 32 - 1


def test_only_frames_beyond_32_bits_are_refused(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o",
                    str(tmp_path / "main")], check=True)
    tiles = [1, 1024, 129600, M // 48, M // 48 + 1, M // 4, M // 4 + 1]
    entries = [0, 1, 100, 300_000, M // 18, M // 18 + 1, 240_000_000, 2 * (M // 3), 2 * ((M + 1) // 3) + 2, M]
    cases = [(t, e) for t in tiles for e in entries]
    out = subprocess.run([str(tmp_path / "main"), *(str(x) for c in cases for x in c)], check=True, capture_output=True,
                         text=True).stdout.split()
    for (t, e), ok, cap in zip(cases, out[::2], out[1::2]):
        least = max(1 << 14, 4 * t, e * 3 // 2)
        assert int(ok) == (least <= M), (t, e)
        if least <= M:
            assert least <= int(cap) <= M, (t, e)
            assert int(cap) == min(M, max(3 << 16, 48 * t, 18 * e))
