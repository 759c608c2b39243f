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


FEW_THREADS = textwrap.dedent("""
    #include "host_pool.h"
    #include <cerrno>
    #include <cstdio>
    #include <dlfcn.h>
    #include <pthread.h>
    namespace msbfs { int host_threads() { return 5; } }
    static std::atomic<int> threads_left{0};
    extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg)
    noexcept {
      if (threads_left.fetch_sub(1) <= 0) return EAGAIN;
      using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
      return reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, arg);
    }
    int main() {
      for (int allowed : {0, 2, 5}) {
        threads_left = allowed;
        msbfs::HostPool pool;
        if (pool.reserve(4) != (unsigned)std::min(allowed, 4)) return 1;
        for (unsigned n : {1u, 5u, 3u}) {
          std::atomic<int> hits[5] = {};
          pool.start(n, [&](unsigned k) { hits[k]++; });
          pool.wait();
          for (unsigned k = 0; k < 5; ++k)
            if (hits[k] != (k < n ? 1 : 0)) return 2;
        }
        std::vector<uint8_t> a(9u << 20, 7);
        msbfs::prefault(pool, a.data(), a.size());
        pool.wait();
        for (uint8_t x : a)
          if (x != 7) return 3;
      }
      puts("ok");
      return 0;
    }
""")


def test_pool_without_enough_threads(tmp_path):
    """Where the system creates no (more) threads, every share still runs
    exactly once and nothing is thrown."""
    (tmp_path / "t.cpp").write_text(FEW_THREADS)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread",
                    f"-I{ROOT / 'webgpu_bfs_gb300' / 'csrc'}", str(tmp_path / "t.cpp"), "-o",
                    str(exe), "-ldl"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stderr)
