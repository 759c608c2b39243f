"""The host worker pool (csrc/host_pool.h), compiled on its own (CPU): jobs of
changing worker counts back to back run every share exactly once, and
prefault leaves what a buffer holds as it is, from any alignment."""
import subprocess
import textwrap
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
SRC = textwrap.dedent("""
    #include "host_pool.h"
    #include <cstdio>
    #include <cstring>
    namespace msbfs { int host_threads() { return 5; } }
    int main() {
      msbfs::HostPool pool;
      unsigned counts[] = {1, 5, 2, 4, 3, 5, 1};
      for (int round = 0; round < 3000; ++round) {
        const unsigned n = counts[round % 7];
        std::atomic<int> hits[5] = {};
        pool.start(n, [&](unsigned k) { hits[k]++; });
        pool.wait();
        for (unsigned k = 0; k < 5; ++k)
          if (hits[k] != (k < n ? 1 : 0)) return 1;
        if (round % 500 == 0)  // past the workers' spin: they sleep
          std::this_thread::sleep_for(std::chrono::milliseconds(2));
      }
      const size_t sizes[] = {1, 4096, (1u << 20) - 1, 1u << 20, (3u << 20) + 17};
      for (size_t bytes : sizes)
        for (size_t off : {size_t(0), size_t(3)}) {
          std::vector<uint8_t> a(bytes + off), b;
          for (size_t i = 0; i < a.size(); ++i) a[i] = (uint8_t)(i * 31 + 7);
          b = a;
          msbfs::prefault(pool, a.data() + off, bytes);
          pool.wait();
          if (a != b) return 2;
        }
      puts("ok");
      return 0;
    }
""")


def test_pool_shares_and_prefault(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread",
                    f"-I{ROOT / 'webgpu_bfs_gb300' / 'csrc'}", str(tmp_path / "t.cpp"), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stderr)
