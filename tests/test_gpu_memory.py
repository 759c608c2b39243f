"""Device memory of the level path (GPU): passes above 16 words are a choice
of speed, so they may not cost a call that a narrower pass has room for."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GB = 1 << 30
FIELDS = ("distance_sum", "eccentricity", "reached")


@pytest.fixture
def torch():
    t = pytest.importorskip("torch")
    yield t
    t.cuda.empty_cache()


@pytest.fixture(scope="module")
def mesh(native):
    """1 M vertices: state of 3.5 GB at 64 words a vertex, 0.9 GB at 16."""
    g = native.generate_erdos_renyi_np(1_000_000, 12 / 999_999, 5)
    src = np.random.default_rng(1).integers(0, g.num_vertices, 2048).astype(np.uint32)
    eng = native.GpuBfsEngine(native.GpuBfsMethod.PushPullAdaptive)
    try:
        eng.set_tuning(max_words_per_pass=16)
        return g, src, eng.run_ms_bfs_stats(g, src)
    finally:
        eng.close()


@contextlib.contextmanager
def _left(torch, free_bytes):
    """The device's memory taken but for about free_bytes."""
    torch.cuda.empty_cache()
    taken = torch.empty(torch.cuda.mem_get_info()[0] - free_bytes, dtype=torch.uint8,
                        device="cuda")
    try:
        yield
    finally:
        taken.untyped_storage().resize_(0)
        torch.cuda.empty_cache()


def test_call_narrows_its_pass_when_memory_is_short(native, torch, mesh):
    g, src, want = mesh
    eng = native.GpuBfsEngine(native.GpuBfsMethod.PushPullAdaptive)
    try:
        eng.upload(g)
        with _left(torch, 2 * GB):
            got = eng.run_ms_bfs_stats(g, src)
        assert all(np.array_equal(got[f], want[f]) for f in FIELDS)
        assert 16 <= eng.last_stats["words_per_vertex"] < 64
    finally:
        eng.close()


def test_wide_state_is_given_back_to_later_calls(native, torch, mesh):
    """A call of 600 sources with rows on the host needs 3 GB of staging, on a
    device with 1 GB free beside the 3.5 GB that a call of 2,048 left in the engine."""
    g, src, want = mesh
    eng = native.GpuBfsEngine(native.GpuBfsMethod.PushPullAdaptive)
    try:
        eng.upload(g)
        with _left(torch, 8 * GB):
            got = eng.run_ms_bfs_stats(g, src)
        assert all(np.array_equal(got[f], want[f]) for f in FIELDS)
        with _left(torch, GB):
            rows = eng.run_ms_bfs(g, src[:600]).reshape(600, -1)
        reached = rows != 0xFFFFFFFF
        assert np.array_equal(reached.sum(1), want["reached"][:600])
        assert np.array_equal(np.where(reached, rows, 0).sum(1, dtype=np.uint64),
                              want["distance_sum"][:600])
    finally:
        eng.close()


def test_tuning_a_small_graph_keeps_the_rule_for_large_ones(native, torch):
    """A graph whose state at 64 words is just beyond an eighth of the device
    memory: 32 words, also on an engine that was tuned on a small graph."""
    total = torch.cuda.mem_get_info()[1]
    V = int(total / 8 / (64 * 4 * 13) * 1.05)
    ring = np.arange(1000, dtype=np.int64)
    big = native.CsrGraph.from_edge_list(
        V, np.concatenate([np.stack([ring, (ring + k) % 1000], 1) for k in range(1, 12)]))
    small = native.generate_graph500_rmat(12, 8, 3)
    src = np.arange(2048, dtype=np.uint32) % 1000
    for tuned in (False, True):
        eng = native.GpuBfsEngine(native.GpuBfsMethod.PushPullAdaptive)
        try:
            if tuned:
                eng.autotune(small, native.sample_sources(small, 1, 2, min_degree=1))
            st = eng.run_ms_bfs_stats(big, src)
            assert (st["reached"] == 1000).all()
            assert eng.last_stats["words_per_vertex"] == 32, tuned
        finally:
            eng.close()
