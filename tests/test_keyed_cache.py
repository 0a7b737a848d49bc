"""The bounded cache of the kernels' tensor maps (host C++): a deep model's maps, asked for in the same order step after step, stay;
other keys push only their own set's oldest out; nothing is ever found under another key."""
import os
import shutil
import subprocess

import pytest

from logssms_b200.ops import build

PROGRAM = r"""
#include <cstdio>
#include "lb200/keyed_cache.h"
typedef lb200::KeyedCache<long, 5, 512, 8> Cache;
int main() {
    Cache c;
    if (c.find({1, 2, 3, 4, 5}) != nullptr) return 1;
    // 66 layers of 6 weights (2 MB apart) and 2 caches, 9 activations of addresses that come in turn, six row counts
    auto step = [&](int rows) {
        int made = 0, wrong = 0;
        auto ask = [&](Cache::Key k) {
            const long want = k[0] * 31 + k[1] * 7 + k[2] + k[3] + k[4];
            const long* v = c.find(k);
            if (v == nullptr) { ++made; c.put(k, want); }
            else if (*v != want) ++wrong;
        };
        for (int layer = 0; layer < 66; ++layer) {
            for (int i = 0; i < 6; ++i) {
                ask({0x7f0000000000l + (layer * 6l + i) * (2 << 20), 1280 + 512 * i, 1280, 1280, 128});
                ask({0x7e0000000000l + ((layer * 6l + i) % 9) * 40960, rows, 1280, 1280, 16});
            }
            for (int i = 0; i < 2; ++i) ask({0x7d0000000000l + (layer * 2l + i) * (64 << 20), 8192, 256, 256, 32});
        }
        if (wrong) std::printf("wrong %d\n", wrong);
        return made;
    };
    int first = step(9), again = step(9), others = 0, back;
    for (int rows = 10; rows < 16; ++rows) others += step(rows);
    back = step(9);
    std::printf("%d %d %d %d\n", first, again, others, back);
    for (long i = 0; i < 100000; ++i) c.put({i * 4096, 1, 2, 3, 4}, i);        // bounded: the last ones are there
    int kept = 0;
    for (long i = 0; i < 100000; ++i) { const long* v = c.find({i * 4096, 1, 2, 3, 4}); if (v != nullptr) { if (*v != i) return 2; ++kept; } }
    std::printf("%d %d\n", kept, c.find({99999l * 4096, 1, 2, 3, 4}) != nullptr);
    return 0;
}
"""


def test_maps_of_a_deep_model_stay(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    source, program = tmp_path / "cache.cpp", str(tmp_path / "cache")
    source.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", build.INCLUDE, "-o", program, str(source)], check=True)
    run = subprocess.run([program], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and "wrong" not in run.stdout, run.stdout
    steps, flood = run.stdout.splitlines()
    # 66 * (6 + 2) weights and caches and 9 activations, made once; other row counts bring 9 activations each
    assert steps.split() == ["537", "0", "54", "0"]
    assert flood.split() == ["4096", "1"]
