"""b200bfs_bfs_noalloc on a caller's own CSR, in any vertex and neighbour
order: depth and levels against the oracle's queue BFS, and a neighbour one
level nearer as every parent, where its frontier list, its direction rule and
its bitmap words have their edges."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _csr(edges, n, rng=None):
    e = edges[edges[:, 0] != edges[:, 1]]
    e = np.unique(np.concatenate([e, e[:, ::-1]]), axis=0)
    if rng is not None:  # neighbours in no order
        e = e[np.lexsort((rng.random(len(e)), e[:, 0]))]
    row_ptr = np.zeros(n + 1, np.int64)
    row_ptr[1:] = np.cumsum(np.bincount(e[:, 0], minlength=n))
    return row_ptr, e[:, 1].astype(np.int32)


def _levels(row_ptr, col, root):
    n = row_ptr.size - 1
    lv = np.full(n, -1, np.int64)
    lv[root] = 0
    front = np.array([root])
    while front.size:
        out = np.concatenate([col[row_ptr[v]:row_ptr[v + 1]] for v in front])
        out = np.unique(out[(out >= 0) & (out < n)])
        out = out[lv[out] < 0]
        lv[out] = lv[front[0]] + 1
        front = out
    return lv


def _check(row_ptr, col, roots):
    import torch
    import b200bfs

    n = row_ptr.size - 1
    d_row, d_col = torch.from_numpy(row_ptr).cuda(), torch.from_numpy(col).cuda()
    d_pred = torch.full((n,), 7, dtype=torch.int64, device="cuda")
    for root in roots:
        depth = b200bfs.bfs_noalloc(d_row.data_ptr(), d_col.data_ptr(), n, int(root),
                                    d_pred.data_ptr(), torch.cuda.current_stream().cuda_stream)
        pred = d_pred.cpu().numpy()
        want = _levels(row_ptr, col, root)
        assert np.array_equal(pred >> 48, want)
        assert depth == want.max() + 1
        parent = pred & ((1 << 48) - 1)
        v = np.nonzero(want > 0)[0]
        assert np.array_equal(want[parent[v]], want[v] - 1)
        for x in v[:: max(1, v.size // 500)]:
            assert parent[x] in col[row_ptr[x]:row_ptr[x + 1]]
        assert parent[root] == root


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 1000, 4097])
def test_random_graphs(built, n):
    rng = np.random.default_rng(n)
    edges = np.stack([(n * rng.random(4 * n) ** 3).astype(np.int64), rng.integers(0, n, 4 * n)], 1)
    row_ptr, col = _csr(edges, n, rng)
    hub = int(np.diff(row_ptr).argmax())
    _check(row_ptr, np.append(col, 0).astype(np.int32), [hub, 0, n - 1])


@pytest.mark.parametrize("scale", [12, 16])
def test_generated_graph_in_its_own_order(built, scale):
    edges = O.generate_edges(scale)
    row_ptr, col = _csr(edges, 1 << scale)
    deg = np.diff(row_ptr)
    _check(row_ptr, col, [int(deg.argmax()), int(np.nonzero(deg)[0][0]), int(np.argmin(deg))])


@pytest.mark.parametrize("leaves", [65535, 65536, 65537, 200000])
def test_list_is_full(built, leaves):
    """Two stars joined at their hubs: the second level has as many rows as the
    frontier list has room for, and more; long enough rows elsewhere keep the
    rule top-down."""
    i = np.arange(leaves)
    edges = np.concatenate([np.stack([np.zeros(leaves, int), i + 1], 1),
                            np.stack([i + 1, leaves + 1 + i], 1)])
    n = 2 * leaves + 1
    m = 40 * leaves  # a second component with most of the entries
    rng = np.random.default_rng(1)
    rest = n + rng.integers(0, 5000, (m, 2))
    row_ptr, col = _csr(np.concatenate([edges, rest]), n + 5000)
    import torch
    import b200bfs

    d_row, d_col = torch.from_numpy(row_ptr).cuda(), torch.from_numpy(col).cuda()
    d_pred = torch.empty(n + 5000, dtype=torch.int64, device="cuda")
    assert b200bfs.bfs_noalloc(d_row.data_ptr(), d_col.data_ptr(), n + 5000, 0,
                               d_pred.data_ptr()) == 3
    pred = d_pred.cpu().numpy()
    want = np.full(n + 5000, -1, np.int64)
    want[0], want[1:leaves + 1], want[leaves + 1:n] = 0, 1, 2
    assert np.array_equal(pred >> 48, want)
    assert np.array_equal(pred[leaves + 1:n] & ((1 << 48) - 1), i + 1)


def test_ids_out_of_range_are_ignored(built):
    rng = np.random.default_rng(5)
    n = 3001
    row_ptr, col = _csr(rng.integers(0, n, (9 * n, 2)), n, rng)
    bad = rng.random(col.size) < 0.05
    keep = col.copy()
    col[bad] = rng.choice([-1, -2**31, n, n + 31, 2**31 - 1], int(bad.sum()))
    # a removed entry's twin goes too, so that the rest stays symmetric
    src = np.repeat(np.arange(n), np.diff(row_ptr))
    gone = set(zip(keep[bad].tolist(), src[bad].tolist()))
    for k in range(col.size):
        if (int(src[k]), int(keep[k])) in gone:
            col[k] = -1
    _check(row_ptr, col, [0, 17, n - 1])


def test_decreasing_row_pointers_are_empty_rows(built):
    """Row v ends before it begins: it has no entries, as root as well.  The
    entries it reaches back over are ignored ids, which the next row has too."""
    rng = np.random.default_rng(6)
    n, v = 2001, 1000
    edges = rng.integers(0, n, (5 * n, 2))
    row_ptr, col = _csr(edges[(edges != v).all(axis=1)], n, rng)
    at = row_ptr[v]
    col = np.concatenate([col[:at], np.full(5, -1, np.int32), col[at:]])
    row_ptr[v:] += 5
    row_ptr[v + 1] -= 5
    assert row_ptr[v + 1] < row_ptr[v]
    _check(row_ptr, col, [v, 0, v - 1, v + 1])


def test_path_and_grid(built):
    i = np.arange(5000)
    row_ptr, col = _csr(np.stack([i[:-1], i[1:]], 1), 5000)
    _check(row_ptr, col, [0, 2500])
    x = np.arange(120 * 77).reshape(120, 77)
    edges = np.concatenate([np.stack([x[:, 1:].ravel(), x[:, :-1].ravel()], 1),
                            np.stack([x[1:].ravel(), x[:-1].ravel()], 1)])
    row_ptr, col = _csr(edges, x.size)
    _check(row_ptr, col, [0, 4321])


def test_calls_of_several_threads(built):
    """Searches of graphs of unlike sizes from four threads at once, each on a
    stream of its own: they share the library's one scratch array."""
    import threading

    import torch
    import b200bfs

    graphs, errors = [], []
    for k in range(4):
        rng = np.random.default_rng(k)
        n = [70001, 300, 9001, 33][k]
        row_ptr, col = _csr(rng.integers(0, n, (6 * n, 2)), n, rng)
        root = int(np.diff(row_ptr).argmax())
        graphs.append((row_ptr, col, root, _levels(row_ptr, col, root)))

    def work(row_ptr, col, root, want):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                d_row, d_col = torch.from_numpy(row_ptr).cuda(), torch.from_numpy(col).cuda()
                d_pred = torch.empty(want.size, dtype=torch.int64, device="cuda")
            for _ in range(100):
                with torch.cuda.stream(stream):
                    d_pred.fill_(7)
                depth = b200bfs.bfs_noalloc(d_row.data_ptr(), d_col.data_ptr(), want.size, root,
                                            d_pred.data_ptr(), stream.cuda_stream)
                assert depth == want.max() + 1
                assert np.array_equal(d_pred.cpu().numpy() >> 48, want)
        except BaseException as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=g) for g in graphs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
