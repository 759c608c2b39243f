"""The traversal's grid barrier when its wait runs out (GPU).

MSBFS_BARRIER_SPINS limits the polls of a barrier. The graph is a star of two
million leaves searched from its hub: one thread writes the hub's queue entries
(milliseconds) while all other blocks poll, far longer than 64 times.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import assert_same

pytestmark = pytest.mark.gpu

TIMEOUT = 4


@pytest.fixture(scope="module")
def star(native):
    return native.star_graph(2_000_001)


@pytest.fixture
def stuck_engine(native, monkeypatch):
    monkeypatch.setenv("MSBFS_BARRIER_SPINS", "64")
    eng = native.GpuBfsEngine(native.GpuBfsMethod.PushPullAdaptive)
    eng.set_tuning(max_words_per_pass=1)
    yield eng
    eng.close()


def _stats_call(native, eng, g, src):
    """(return code, statistics of the call)."""
    st = native.Stats()
    out = np.zeros(len(src), native.SOURCE_STATS_DTYPE)
    dg = eng.upload(g)
    lib = native._native.lib()
    rc = lib.msbfs_run_ms_bfs_stats(eng._h, dg.handle, src.ctypes.data_as(C.POINTER(C.c_uint32)),
                                    src.size, out.ctypes.data_as(C.c_void_p), C.byref(st))
    return rc, st.as_dict()


def test_no_level_runs_on_a_stuck_workspace(native, stuck_engine, star):
    """The block that comes late does not open the barrier that the others left,
    nor do the passes queued behind: the sources are all that is reached."""
    for passes in (1, 3):
        rc, st = _stats_call(native, stuck_engine, star, np.zeros(32 * passes, np.uint32))
        assert rc == TIMEOUT and st["passes"] == passes
        assert st["reached_pairs"] == 32 * passes and st["levels"] == 1


def test_stuck_call_is_reported_after_later_calls(native, stuck_engine, star):
    """Asynchronous calls behind the stuck one, on the same workspace and on
    the one-block-per-source path: the next synchronise reports it, once."""
    torch = pytest.importorskip("torch")
    small = native.Grid2D(20, 20)
    out = torch.empty(star.num_vertices, dtype=torch.int32, device="cuda")
    rows = torch.empty((2, 400), dtype=torch.int32, device="cuda")
    cta = native.GpuBfsMethod.WorkgroupPersistentBfs
    eng, src = stuck_engine, np.array([0, 399], np.uint32)
    eng.run_ms_bfs_device(star, src[:1], out.data_ptr())
    eng.run_ms_bfs_device(star, src[:1], out.data_ptr())
    eng.run_ms_bfs_device(small.graph, src, rows.data_ptr(), method=cta)
    with pytest.raises(native.BfsError) as ei:
        eng.synchronize()
    assert ei.value.code == TIMEOUT
    # the engine stays usable: the same path driven from the host, and the other
    eng.run_ms_bfs_device(small.graph, src, rows.data_ptr(), method=cta)
    eng.synchronize()
    assert_same(rows.cpu().numpy().view(np.uint32).ravel(), small.ms_bfs_oracle(src))
    eng.set_profiling(3)
    want = np.ones(star.num_vertices, np.uint32)
    want[0] = 0
    assert_same(eng.run_ms_bfs(star, src[:1]), want, star, src[:1])
