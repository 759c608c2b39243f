"""Launches whose shared-memory limits another object of the process also
sets (GPU): the limit belongs to the kernel, so objects of different size
must not take it from one another."""
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
