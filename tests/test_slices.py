"""The split of a segment list over a launch's blocks (pb_slices.h), on the host.

Every block's loop has to end and every segment to be taken by one block, for
lists of any length and grids of any height: an empty list above all, which the
energy windows of the bremsstrahlung scorer leave where every electron lies in
one of them.
"""

import shutil
import subprocess
from pathlib import Path

import pytest

HEADER = Path(__file__).resolve().parents[1] / "pyrite_b200" / "csrc" / "pb_slices.h"

SOURCE = r"""
#include <cstdio>
#include <vector>
#include "%s"
int main() {
    long long bad = 0;
    for (int most : {64, 256})
        for (int64_t ny : {1, 2, 3, 17, 74, 148, 444}) {
            std::vector<int64_t> lives = {0, 1, 2, 63, 64, 65, 255, 256, 257, 511, 513, 1000, 82000};
            for (int64_t g : {ny - 1, ny, ny + 1, most * ny - 1, most * ny, most * ny + 1, 2 * most * ny + 1}) lives.push_back(g);
            for (int64_t live : lives)
                for (int dealt = 0; dealt < 2; ++dealt) {
                    std::vector<int> seen(live, 0);
                    for (int64_t y = 0; y < ny; ++y) {
                        const pb::SegSlice s = pb::seg_slice(live, y, ny, most, dealt);
                        bool ok = s.chunk >= 1 && s.chunk <= most && s.step >= s.chunk && s.begin >= 0 && s.end <= live;
                        if (live == 0) ok = ok && s.begin >= s.end;
                        if (!ok) {
                            std::printf("live %%lld y %%lld ny %%lld dealt %%d: begin %%lld end %%lld step %%lld chunk %%lld\n",
                                        (long long)live, (long long)y, (long long)ny, dealt, (long long)s.begin,
                                        (long long)s.end, (long long)s.step, (long long)s.chunk);
                            ++bad;
                            continue;
                        }
                        for (int64_t c = s.begin; c < s.end; c += s.step)
                            for (int64_t j = c; j < s.end && j < c + s.chunk; ++j) ++seen[j];
                    }
                    for (int64_t j = 0; j < live; ++j) bad += seen[j] != 1;
                }
        }
    std::printf("%%lld\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_every_segment_once_and_every_loop_ends(tmp_path):
    src, exe = tmp_path / "slices.cc", tmp_path / "slices"
    src.write_text(SOURCE % HEADER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "0", r.stdout
