"""Grid rule of the CTA path's global-bitmap mode (csrc/cta_grid.h), compiled
on its own (CPU): whole rounds within the SM share that a server gives a slot."""
import subprocess
import textwrap
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
SRC = textwrap.dedent("""
    #include "cta_grid.h"
    #include <cstdio>
    int main() {
      // road 1448 x 1448: 456 resident blocks, bitmaps of 304 in the L2
      for (int share : {100, 85, 50, 30, 1})
        for (size_t S : {1, 65, 160, 304, 400, 456, 512, 700, 1024, 2048})
          printf("%d %zu %zu\\n", share, S, msbfs::global_bitmap_grid(456 * share / 100, 304, S));
    }
""")


def test_rounds_fit_the_share(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT / 'webgpu_bfs_gb300' / 'csrc'}",
                    str(tmp_path / "t.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    grids = {tuple(map(int, l.split()[:2])): int(l.split()[2]) for l in out.splitlines()}
    for (share, S), blocks in grids.items():
        resident = 456 * share // 100
        assert 1 <= blocks <= min(resident, S)
        rounds = -(-S // blocks)
        assert blocks == -(-S // rounds)  # no round nearly empty
    # one round as long as the share holds the sources' blocks, as at 100%
    assert [grids[85, S] for S in (160, 304)] == [grids[100, S] for S in (160, 304)] == [160, 304]
    assert grids[100, 512] == grids[85, 512] == 256
    assert grids[100, 400] == 400 and grids[85, 400] == 200
