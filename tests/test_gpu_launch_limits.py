"""Launches whose shared-memory limits another object of the process also
sets (GPU): the limit belongs to the kernel, so objects of different size
must not take it from one another."""
import threading

import numpy as np
import pytest

from conftest import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alg", [0, 1])
def test_batches_of_different_size_alive_at_once(native, tmp_path, alg):
    """A batch at the vertex limit runs after a tiny one was created, as
    bit-parallel (0) and as single-source (1) items."""
    grid = native.Grid2D(512, 512)  # MSBFS_BATCH_MAX_VERTICES vertices
    src = np.array([0, 513 * 200, 512 * 512 - 1], np.uint32)
    star, hub = native.star_graph(9), np.array([0], np.uint32)
    big = native.BatchedBfs([(grid.graph, src)])
    small = native.BatchedBfs([(star, hub)])
    try:
        for k, b in enumerate((big, small)):
            cache = tmp_path / f"{k}.txt"
            cache.write_text(f"{b.config(0)['class']} {alg} 1 16 1 0 1.0\n")
            b.autotune(samples_per_class=1, cache_path=str(cache))
        for _ in range(2):
            big.run()
            small.run()
        assert_same(big.result(0), grid.ms_bfs_oracle(src), grid.graph, src, f"alg={alg}")
        assert_same(small.result(0), [0] + [1] * 8, star, hub, f"alg={alg}")
    finally:
        small.close()
        big.close()

def test_cta_calls_of_different_size_from_two_threads(native):
    """One-source calls on a tree of 40,000 vertices (seven levels, so many
    calls) and on a 1,000 x 1,200 grid, each from a thread with an engine of
    its own: one kernel, with 37 KB and 183 KB of shared memory."""
    n = 40_000
    v = np.arange(1, n)
    up = np.stack([v, (v - 1) // 7], 1)
    tree = native.CsrGraph.from_edge_list(n, np.concatenate([up, up[:, ::-1]]))
    w, h = 1000, 1200
    grid = native.Grid2D(w, h).graph
    done = threading.Event()
    failures = []

    def serve(g, calls, ecc):
        eng = native.GpuBfsEngine(native.GpuBfsMethod.WorkgroupPersistentBfs)
        try:
            for _ in range(calls):
                st = eng.run_ms_bfs_stats(g, [0])[0]
                assert st["reached"] == g.num_vertices and st["eccentricity"] == ecc
                if done.is_set():
                    break
        except Exception as e:
            failures.append(f"V={g.num_vertices}: {e}")
        finally:
            eng.close()

    small = [threading.Thread(target=serve, args=(tree, 10 ** 9, 6)) for _ in range(2)]
    for t in small:
        t.start()
    serve(grid, 400, w + h - 2)
    done.set()
    for t in small:
        t.join()
    assert not failures, failures
