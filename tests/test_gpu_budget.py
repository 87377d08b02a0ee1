"""Engines with a device-memory budget: what a call needs beside a prepared
graph is its own buffers only.  The smallest budget of a sequence of calls is
found by bisection."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEP = 4096
IDS = 1 << 16  # of pred and levels, at least

# a graph of few rows: pred and its map outweigh what the build needs
EDGES = np.random.default_rng(1).integers(0, 5000, (20000, 2))


def _fits(budget, calls, flags=0, option=None, edges=EDGES):
    import b200bfs

    e = b200bfs.Engine(0, budget)
    try:
        if option:
            e.set_option(*option)
        e.build_from_edges(edges, flags=flags)
        for call in calls:
            call(e)
        return True
    except b200bfs.B200BfsError as x:
        if x.code != 3:  # B200BFS_ERR_OOM
            raise
        return False
    finally:
        e.close()


def _smallest(calls, **how):
    lo, hi = 0, 1 << 18
    while not _fits(hi, calls, **how):
        lo, hi = hi, 2 * hi
    while hi - lo > STEP:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if _fits(mid, calls, **how) else (mid, hi)
    return hi


def _prepare(e):
    e.prepare(16)


def _search(e):
    e.run(int(e.find_roots(1)[0]), 16)


def _levels(e):
    e.get_levels()


def _batch(e):
    e.run_batch([int(r) for r in e.find_roots(64)])


def test_levels_beside_a_prepared_graph(built):
    """4 bytes per id; the one-kernel search's own buffers, which fit until
    then, give way."""
    base = _smallest([_prepare])
    assert _fits(base + 4 * IDS + STEP, [_prepare, _search, _levels])


@pytest.mark.parametrize("flags", [0, 3])
def test_batch_beside_a_prepared_graph(built, flags):
    """As much as with the one-kernel search switched off."""
    budget = _smallest([_prepare, _batch], flags=flags, option=("persistent", 0))
    assert _fits(budget, [_prepare, _search, _batch], flags=flags)


def test_validation_of_a_callers_pred(built):
    """With CoreBFS as much as that of the engine's own: pred and its depth map
    are one array."""
    def validate(e):
        assert e.validate(e.root)[0] == 0

    def validate_pred(e):
        assert e.validate_pred(e.root, e.pred, corebfs=True)[0] == 0

    def search(e):
        e.root = int(e.find_roots(1)[0])
        e.run(e.root, 16)
        e.pred = e.get_pred()

    budget = _smallest([_prepare, search, validate], flags=1)
    assert _fits(budget + STEP, [_prepare, search, validate_pred], flags=1)


def test_sorting_long_rows_takes_no_more_than_the_entries(built):
    """300 hubs of 16,500 entries among 4 M vertices: their bitmaps together
    would take four times the entries."""
    rng = np.random.default_rng(1)
    hubs, length, n = 300, 16500, 4000000
    leaf = hubs + rng.integers(0, n - hubs, hubs * length)
    leaf[:n - hubs] = np.arange(hubs, n)
    edges = np.stack([np.repeat(np.arange(hubs), length), leaf], 1)
    # 8 bytes per edge for the edges, for their entries and for what they are
    # compacted to (or the bitmaps), and six arrays per id: 36 bytes
    assert _fits(24 * len(edges) + 36 * 2**22, [], edges=edges)


def test_searches_go_on_without_the_one_kernel(built):
    """After its buffers gave way the level loop searches; with room again the
    next prepare brings them back."""
    import b200bfs

    budget = _smallest([_prepare]) + 4 * IDS + STEP
    e, free = b200bfs.Engine(0, budget), b200bfs.Engine(0)
    for x in (e, free):
        x.build_from_edges(EDGES)
        x.prepare(16)
    roots = [int(r) for r in e.find_roots(3)]
    launches = []
    for r in roots + roots:
        assert np.array_equal(e.run(r), free.run(r))
        launches.append(e.run_stats().kernel_launches)
        assert np.array_equal(e.get_levels(), free.get_levels())
        assert e.validate(r) == free.validate(r)
    assert launches[0] == 1 and min(launches[1:]) > 1
    e.prepare(16)
    e.run(roots[0])
    assert e.run_stats().kernel_launches == 1
    e.close()
    free.close()
