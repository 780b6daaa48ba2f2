"""Which entries of its distance-bias table the tcgen05 attention kernel reads, over portions that end next to their line's end: the
kernel's own index function, compiled for the host."""
import glob
import shutil
import subprocess

import pytest

from neuronx_distributed_llama3_2_b200.ops import _lib

# the tiles that the kernel visits without a mask (128 query rows of four warps, 64 keys), restated
PROGRAM = r"""
#include "score_mod.cuh"
int main() {
    long long read = 0, clamped = 0;
    const int windows[] = {0, 64, 100, 300}, keeps[] = {0, 70}, capacities[] = {64, 70, 128, 200, 448};
    for (int window : windows) for (int keep : keeps) for (int rows : capacities)
        for (int tokens = 1; tokens <= 300; tokens += 13) for (int start = 0; start + tokens <= rows; start += 7) {
            const int end = start + tokens;
            const int entries = window > 0 && window < rows && keep == 0 ? window : rows;
            for (int m0 = 0; m0 < tokens; m0 += 128) for (int warp = 0; warp < 4; ++warp) for (int n0 = 0; n0 < end; n0 += 64) {
                const int first = m0 + warp * 32 + start, last = first + 31;       // positions of the warp's rows
                if (n0 + 64 > end || n0 + 63 > first || (window > 0 && last - window + 1 > n0 && n0 + 64 > keep)) continue;
                for (int r = 0; r < 32; ++r) {
                    const int d0 = first + r - n0, at = score::table_entry(d0, entries);
                    if (at - 63 < 0 || at >= entries) return 2;                      // outside the table
                    if (m0 + warp * 32 + r < tokens && at != d0) return 3;           // a real row reads its own distances
                    ++read, clamped += at != d0;
                }
            }
        }
    return read > 0 && clamped > 0 ? 0 : 4;                                          // there are rows that need the clamp
}
"""


def test_unmasked_tiles_read_inside_the_table(tmp_path):
    if not (shutil.which(_lib._nvcc()) or glob.glob(_lib._nvcc())):
        pytest.skip("needs nvcc")
    (tmp_path / "index.cu").write_text(PROGRAM)
    subprocess.run([_lib._nvcc(), "-std=c++17", "-I", _lib.CSRC_DIR, "-I", _lib.INCLUDE_DIR, "-o", str(tmp_path / "index"),
                    str(tmp_path / "index.cu")], check=True)
    assert subprocess.run([str(tmp_path / "index")]).returncode == 0
