"""The budget network's workspace: room made for a batch holds the partial sums of every
smaller batch (hrnn_b200/csrc/mlp_ranges.hpp, compiled for the host)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include "mlp_ranges.hpp"
int main() {
    size_t n = 0, n3 = 0;  // the most of any batch so far
    for (int B = 1; B <= (1 << 20); B += B < 20000 ? 1 : 997) {
        const hrnn::Ranges r(B);
        if ((size_t)r.per * r.n < (size_t)B || (size_t)r.per3 * r.n3 < (size_t)B)
            return std::printf("%d rows are not all in a range\n", B), 1;
        n = r.n > n ? r.n : n;
        n3 = r.n3 > n3 ? r.n3 : n3;
        const hrnn::MostRanges room(B);
        if (room.n < n || room.n3 < n3)
            return std::printf("room for %d rows: %zu and %zu ranges, a smaller batch has %zu and %zu\n", B, room.n,
                               room.n3, n, n3), 1;
    }
    return 0;
}
"""


def test_room_for_a_batch_holds_every_smaller_one(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("needs g++")
    src, exe = tmp_path / "ranges.cpp", str(tmp_path / "ranges")
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "hrnn_b200", "csrc"), str(src), "-o", exe],
                   check=True)
    p = subprocess.run([exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout
