"""The one-kernel search (option "persistent" 2, 3 and 4) against the level loop
(0) and the oracle: levels, auto_tuning_data, run statistics, per-level
records and validity of parents, on graphs whose sizes, frontiers and depths
sit at its limits."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

KEYS = ("levels", "num_td_levels", "num_bu_levels", "bu_level_mask", "visited", "edges_scanned_td",
        "edges_scanned_bu", "td_bytes", "bu_bytes", "pred_bytes")


@pytest.fixture(scope="module")
def engine(built):
    import b200bfs

    e = b200bfs.Engine(0)
    yield e
    e.close()


def _search(engine, mode, root, alpha, beta):
    engine.set_option("persistent", mode)
    try:
        at = engine.run(root, 16, alpha, beta)
    finally:
        engine.set_option("persistent", 1)
    st = engine.run_stats()
    return ([int(x) for x in at], {k: getattr(st, k) for k in KEYS},
            [{k: v for k, v in x.items() if k != "ms"} for x in engine.level_stats()])


def _compare(engine, g, roots, alpha=10.0, beta=14.0, modes=(2, 3, 4), corebfs=False):
    engine.prepare(16, alpha, beta)
    engine.run(int(roots[0]), 16, alpha, beta)  # the first search fills pred once
    for r in (int(r) for r in roots):
        want = _search(engine, 0, r, alpha, beta)
        levels = engine.get_levels()
        if not corebfs:
            assert np.array_equal(levels[: g.nverts], g.levels(r))
        verdict = engine.validate(r)
        assert verdict[0] == 0 or want[1]["visited"] == 1  # a root without edges
        for mode in modes:
            assert _search(engine, mode, r, alpha, beta) == want, (mode, r)
            st = engine.run_stats()
            assert st.kernel_launches <= 2 and st.device_ms > 0 and st.td_ms > 0
            assert np.array_equal(engine.get_levels(), levels), (mode, r)
            assert engine.validate(r) == verdict


@pytest.mark.parametrize("scale,flags", [(5, 0), (10, 0), (10, 3), (14, 1), (16, 2), (18, 0)])
@pytest.mark.parametrize("alpha,beta", [(10.0, 14.0), (1e-9, 14.0), (1e9, 14.0), (30.0, 2.0),
                                        (1e-15, 14.0), (30.0, 1e-16)])
def test_generated_graphs(engine, scale, flags, alpha, beta):
    """Every direction sequence: the rule, all top-down (alpha 1e-9),
    bottom-up after level 1 (1e9), an early return to top-down, and limits of
    the switch beyond 64 bits."""
    edges = O.generate_edges(scale)
    g = O.Graph(edges)
    engine.generate_graph(scale, 16, flags=flags)
    has = engine.has_edge_all()[: g.nverts]
    roots = list(np.nonzero(has)[0][[0, -1]]) + list(np.nonzero(has == 0)[0][:1])
    _compare(engine, g, roots, alpha, beta, corebfs=bool(flags & 1))


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 127, 130, 300, 1000])
def test_paths(engine, n):
    """One row per level; beyond 64 levels the records come from the second
    buffer."""
    edges = np.stack([np.arange(n - 1), np.arange(1, n)], axis=1).astype(np.int64)
    engine.build_from_edges(edges)
    _compare(engine, O.Graph(edges), [0, n // 2, n - 1])


@pytest.mark.parametrize("leaves", [1, 30, 31, 32, 33, 127, 128, 129, 1000, 40000])
def test_stars(engine, leaves):
    """A frontier of rows of one entry, as many as lie in a lookup window and
    more, expanded top-down (alpha 1e-9) and bottom-up."""
    i = np.arange(leaves)
    edges = np.concatenate([np.stack([np.zeros(leaves, int), i + 1], 1),
                            np.stack([i + 1, leaves + 1 + i], 1)]).astype(np.int64)
    engine.build_from_edges(edges)
    for alpha in (10.0, 1e-9):
        _compare(engine, O.Graph(edges), [0, leaves + 1, 1], alpha)


@pytest.mark.parametrize("seed", range(4))
def test_ragged_degrees(engine, seed):
    """Skewed degrees, duplicates, self-loops and several components."""
    rng = np.random.default_rng(seed)
    n, m = 40000 + 7 * seed, 150001
    edges = np.stack([(n * rng.random(m) ** 3).astype(np.int64), rng.integers(0, n, m)], axis=1)
    engine.build_from_edges(edges)
    g = O.Graph(edges)
    hub = int(np.bincount(edges.ravel()).argmax())
    roots = [hub] + [int(r) for r in O.find_roots(g.has_edge(), n, 3)]
    for alpha in (10.0, 1e-9, 1e9):
        _compare(engine, g, roots, alpha)


def test_forms_keep_the_level_loop(engine):
    """An option that picks a form of the level loop takes the search there."""
    engine.generate_graph(12, 16)
    engine.prepare(16)
    root = int(engine.find_roots(1)[0])
    engine.run(root)
    assert engine.run_stats().kernel_launches == 1
    for name, value, default in (("bu_kernel", 3, 2), ("td_kernel", 7, 4), ("bu_spec", 0, 1)):
        engine.set_option(name, value)
        engine.run(root)
        assert engine.run_stats().kernel_launches > 2
        engine.set_option(name, default)


def test_engines_of_two_threads(built):
    """Searches of two engines at once, on their own streams: cooperative
    grids that each need the whole device."""
    import threading

    import b200bfs

    def work(scale, out):
        e = b200bfs.Engine(0)
        e.generate_graph(scale, 16)
        e.prepare(16)
        roots = [int(r) for r in e.find_roots(4)]
        for i in range(60):
            r = roots[i % 4]
            e.run(r)
            lv = e.get_levels()
            out.append(np.array_equal(lv, out[i % 4][0]) if i >= 4 else (lv, e.validate(r)[0]))
        e.close()

    results = [[], []]
    threads = [threading.Thread(target=work, args=(18 + k, results[k])) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for out in results:
        assert len(out) == 60 and all(o[1] == 0 for o in out[:4]) and all(out[4:])
