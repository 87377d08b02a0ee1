"""CSR construction around the row lengths where its passes change: rows cut
into pieces (2048, pieces of 4096 entries); rows sorted by a warp (up to 256),
by a block (512, 2048, 8192, 16384), by bitmap (above 16384, from R / 512) and
by the segmented sort (between the two); with duplicates and self-loops, plain,
group-reordered and with CoreBFS."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(built):
    import b200bfs

    e = b200bfs.Engine(0)
    yield e
    e.close()


def _edges(degree, n, seed):
    """A hub with `degree` entries before de-duplication, a second one with
    half of them, a ring (nobody is pruned) and a tail of three."""
    rng = np.random.default_rng(seed)
    ring = np.stack([np.arange(n), (np.arange(n) + 1) % n], 1)
    hub = np.stack([np.full(degree, n), rng.integers(0, n, degree)], 1)
    half = np.stack([rng.integers(0, n, degree // 2), np.full(degree // 2, n + 1)], 1)
    loops = np.stack([np.full(3, n), np.full(3, n)], 1)
    tail = np.array([[n, n + 2], [n + 2, n + 3], [n + 3, n + 4]])
    edges = np.concatenate([ring, hub, half, loops, tail]).astype(np.int64)
    return edges[rng.permutation(len(edges))]


@pytest.mark.parametrize("degree", [30, 31, 62, 63, 126, 127, 254, 255, 510, 511, 2045, 2046, 2047, 4094, 4095, 8189, 8190, 8191, 8192, 12287, 16381, 16382, 16383,
                                    40000, 200000])
@pytest.mark.parametrize("flags", [0, 2, 3])
def test_rows(engine, degree, flags):
    import b200bfs

    n = 30000
    edges = _edges(degree, n, degree)
    engine.build_from_edges(edges, flags=flags)
    row_ptr, col, inv, mdeg = (a.astype(np.int64) for a in engine.get_csr())
    e = edges[edges[:, 0] != edges[:, 1]]
    raw = np.bincount(e.ravel(), minlength=n + 5)
    if flags & b200bfs.BUILD_COREBFS:
        e = e[(e < n + 2).all(axis=1)]
    both = np.unique(np.concatenate([e, e[:, ::-1]]), axis=0)
    rows = np.unique(both[:, 0])
    assert np.array_equal(np.sort(inv), rows)
    deg = np.bincount(both[:, 0], minlength=n + 5)
    assert np.array_equal(np.diff(row_ptr), deg[inv])
    if flags & b200bfs.BUILD_COREBFS:
        assert np.array_equal(mdeg, deg[inv])
    else:
        assert np.array_equal(mdeg, raw[inv])
    # the same neighbours, highest degree before de-duplication first
    src = np.repeat(inv, np.diff(row_ptr))
    got = np.stack([src, inv[col]], 1)
    assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], both)
    d = raw[inv[col]]
    inside = np.ones(col.size, bool)
    inside[row_ptr[:-1]] = False
    assert (d[1:][inside[1:]] <= d[:-1][inside[1:]]).all()


def test_complete_graph(engine):
    """9000 vertices: every row is of the longest that a block sorts."""
    n = 9000
    a, b = np.triu_indices(n, 1)
    engine.build_from_edges(np.stack([a, b], 1).astype(np.int64))
    row_ptr, col, inv, _ = engine.get_csr()
    assert np.array_equal(np.diff(row_ptr), np.full(n, n - 1))
    c = col.reshape(n, n - 1)
    want = np.arange(n - 1)[None, :] + (np.arange(n - 1)[None, :] >= np.arange(n)[:, None])
    assert np.array_equal(c, want)


def _same(engine, edges, n):
    """The CSR of a list without self-loops, entry by entry, and its order."""
    engine.build_from_edges(edges)
    row_ptr, col, inv, mdeg = (a.astype(np.int64) for a in engine.get_csr())
    raw = np.bincount(edges.ravel(), minlength=n)
    want = np.unique(np.concatenate([edges[:, 0] * n + edges[:, 1],
                                     edges[:, 1] * n + edges[:, 0]]))
    src = np.repeat(inv, np.diff(row_ptr))
    assert np.array_equal(np.sort(src * n + inv[col]), want)
    assert np.array_equal(mdeg, raw[inv]) and (np.diff(mdeg) <= 0).all()
    # row ids are in the order of the degrees, so every row is ascending
    inside = np.ones(col.size, bool)
    inside[row_ptr[:-1]] = False
    assert (col[1:] > col[:-1])[inside[1:]].all()
    return raw


def test_more_bitmap_rows_than_a_batch(engine):
    """150 rows of 16,500 entries, and room for the bitmaps of 132 (four bytes
    per entry, an eighth of a byte per row of the graph)."""
    rng = np.random.default_rng(2)
    hubs, length, n = 150, 16500, 1200000
    leaf = hubs + rng.integers(0, n - hubs, hubs * length)
    leaf[:n - hubs] = np.arange(hubs, n)
    edges = np.stack([np.repeat(np.arange(hubs), length), leaf], 1)
    raw = _same(engine, edges[rng.permutation(len(edges))], n)
    assert (raw > 16384).sum() * (n // 8) > 4 * raw.sum()


def test_segmented_rows(engine):
    """9 M rows, so that bitmaps begin at 17,578 entries: rows on both sides of
    that and of a block's 16,384, among rows of one to a few entries."""
    rng = np.random.default_rng(3)
    n = 9000000
    lengths = [16383, 16384, 16385, 16500, 17000, 17576, 17577, 17578, 17579, 20000]
    pairs = rng.permutation(np.arange(len(lengths), n)).reshape(-1, 2)
    hubs = [np.stack([np.full(k, h), rng.integers(len(lengths), n, k)], 1)
            for h, k in enumerate(lengths)]
    edges = np.concatenate([pairs] + hubs)
    raw = _same(engine, edges[rng.permutation(len(edges))], n)
    assert ((raw > 16384) & (raw < n // 512)).sum() == 5
