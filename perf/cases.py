"""What this framework's users have it do, as cases that can be timed.

A case names a kind of work and its sizes:

  search    a Graph500 benchmark run: one search after the other from a list of
            roots on a graph that stays resident, as the driver's loop over
            its search keys does, then the levels of the last one in host memory
  batch     one multi-source traversal from up to 64 roots, the deepest level
            of every root, and the levels of some or all of them in host memory
  validate  a search followed by the Graph500 checks of its result
  first     from an edge list (generated, or the caller's in host memory) to
            the CSR in host memory and the first search's levels: what a new
            graph costs
  noalloc   the allocation-free search on a CSR and an output array that the
            caller holds on the device

Parents are not unique, so what is compared is what every correct search
gives: the levels of every vertex, the switch record (auto_tuning_data), the
number of vertices reached, the validator's verdict and its edge count. All of
it is whole numbers and has to be the same.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "graph500-bfs_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import b200bfs  # noqa: E402

# Seeds 2 and 3 are the benchmark's own; further graphs move the second one.
_SEED1 = b200bfs.USERSEED1


def _case(name, kind, scale, **more):
    c = {"kind": kind, "scale": scale, "edgefactor": 16, "corebfs": False, "group": False,
         "roots": 1, "alpha": b200bfs.DEFAULT_ALPHA, "beta": b200bfs.DEFAULT_BETA,
         # vertices and edges of a caller's own edge list, in place of the generator (0)
         "verts": 0, "edges": 0, "fetch": 1}
    if name:
        c["name"] = name
    c.update(more)
    return c


def listed():
    return [
        # one query on a graph that fits in any cache: latency and launches
        # (beta 2, as the -A tuner picks small ones on small graphs)
        _case("search_s12", "search", 12, beta=2.0),
        # one query on the smallest graph of the serving workload, as the
        # headline options (-C, group reordering) build it
        _case("search_s16_core", "search", 16, corebfs=True, group=True, beta=2.0),
        # a short benchmark run on a graph that fits in L2
        _case("search_s20_r4", "search", 20, roots=4),
        # a caller's own edge list: ragged sizes, not a Kronecker graph
        _case("search_own_300007", "search", 19, verts=300007, edges=1900001, roots=3),
        # the serving workload's denser SCALE 22 graph
        _case("search_s22_ef32_r8", "search", 22, edgefactor=32, group=True, roots=8),
        # the SCALE 24 configuration with CoreBFS and the -A tuner's alpha and beta
        _case("search_s24_core_r16", "search", 24, corebfs=True, group=True, roots=16,
              alpha=24.5, beta=20.0),
        # the headline configuration with 16 of its search keys, at the largest
        # scale of which several graphs fit on the device
        _case("search_s26_core_r16", "search", 26, corebfs=True, group=True, roots=16,
              alpha=24.5, beta=20.0),
        # a batch that is not full, every root's levels wanted
        _case("batch_s18_r33", "batch", 18, roots=33, alpha=b200bfs.BATCH_ALPHA, fetch=33),
        # a full batch, where only a few roots' levels are looked at
        _case("batch_s24_r64", "batch", 24, roots=64, alpha=b200bfs.BATCH_ALPHA, fetch=2),
        # search and validation, as the driver does for every validated root
        _case("validate_s23", "validate", 23),
        # a graph that is added to a server: generated, built, searched
        _case("first_s22_core", "first", 22, corebfs=True, group=True),
        # a program that owns the device memory calls the allocation-free
        # search on a CSR of its own, in its own vertex order
        _case("noalloc_s20", "noalloc", 20),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "batch", "validate", "first", "noalloc"])
    top = {"search": 25, "batch": 23, "validate": 22, "first": 20, "noalloc": 19}[kind]
    c = _case(None, kind, rng.randint(12, top))
    c["edgefactor"] = rng.choice([8, 11, 16, 16, 19, 24, 32]) if c["scale"] < 23 else 16
    c["group"] = rng.random() < 0.5
    c["corebfs"] = rng.random() < 0.5
    if kind in ("search", "first") and rng.random() < 0.35:
        c["verts"] = _log_uniform(rng, 1001, 1500007) | 1
        c["edges"] = c["verts"] * rng.randint(5, 20) + rng.randint(1, 9)
        c["scale"] = max(1, (c["verts"] - 1).bit_length())
        # a ragged list's 2-core may be empty or need more than 32 rounds
        c["corebfs"] = False
    if kind == "search":
        c["roots"] = rng.choice([1, 2, 3, 5, 8])
    if kind == "batch":
        c["roots"] = rng.choice([1, 7, 31, 33, 50, 63, 64])
        c["fetch"] = min(c["roots"], rng.choice([1, 2, 3]))
        c["alpha"] = float(rng.choice([10, 30, 100, 200]))
    else:
        c["alpha"] = rng.choice([8.0, 10.0, 24.5])
    c["beta"] = rng.choice([10.0, 14.0, 20.0] if c["scale"] >= 20 else [1.0, 2.0])
    if kind == "noalloc":
        c["corebfs"] = c["group"] = False
    return c


def _own_edges(case, seed):
    """A caller's edge list: skewed degrees, some self-loops and duplicates, ids in no order."""
    rng = np.random.default_rng(seed)
    n, m = case["verts"], case["edges"]
    a = (n * rng.random(m) ** 2).astype(np.int64)
    b = rng.integers(0, n, m)
    ids = rng.permutation(n)
    edges = np.stack([ids[a], ids[b]], axis=1)
    edges[0] = (n - 1, 0)  # the id range is the same for every seed
    return edges


def _flags(case):
    return ((b200bfs.BUILD_COREBFS if case["corebfs"] else 0)
            | (b200bfs.BUILD_GROUP_REORDER if case["group"] else 0))


def _build(eng, state):
    case = state["case"]
    if case["verts"]:
        eng.build_from_edges(state["edges"], 0, _flags(case))
    else:
        eng.generate_graph(case["scale"], case["edgefactor"], _SEED1, state["seed2"], _flags(case))


class _State(dict):
    """A state that gives its engine's device memory back when it goes."""

    def __del__(self):
        if "eng" in self:
            self["eng"].close()


def _own_csr(eng, case, seed2):
    """The symmetric CSR of a generated graph over all 2^scale ids, in the generator's vertex order."""
    n = 1 << case["scale"]
    e = torch.from_numpy(eng.generate_edges(case["scale"], 0, case["edgefactor"] * n, _SEED1, seed2)).cuda()
    e = e[e[:, 0] != e[:, 1]]
    key = torch.unique(torch.cat([e[:, 0] * n + e[:, 1], e[:, 1] * n + e[:, 0]]))
    row_ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    row_ptr[1:] = torch.bincount(key // n, minlength=n).cumsum(0)
    return row_ptr, (key % n).to(torch.int32)


def _pinned(n, dtype):
    return torch.zeros(n, dtype=dtype, pin_memory=True)


def prepare(case, seed):
    state = _State(case=dict(case), seed2=b200bfs.USERSEED2 + seed)
    eng = state["eng"] = b200bfs.Engine(device=0)
    if case["kind"] == "noalloc":
        state["row_ptr"], state["col"] = _own_csr(eng, case, state["seed2"])
        state["pred"] = torch.empty(state["row_ptr"].numel() - 1, dtype=torch.int64, device="cuda")
        degree = state["row_ptr"].diff()
        with_edges = degree.nonzero().flatten()
        state["root"] = int(with_edges[random.Random(seed).randrange(with_edges.numel())])
        return state
    if case["verts"]:
        state["edges"] = _own_edges(case, seed)
    _build(eng, state)
    state["keys"] = [int(r) for r in eng.find_roots(case["roots"], 0, seed % 1000)]
    # results are read back into pinned memory, as the benchmark does
    n = eng.info().pred_size
    state["levels"] = _pinned(n * (case["fetch"] if case["kind"] == "batch" else 1), torch.int32)
    if case["kind"] == "first":
        # room for the CSR of any graph of this size
        m = case["edges"] or case["edgefactor"] << case["scale"]
        state["csr"] = [_pinned(n + 1, torch.int64), _pinned(2 * m, torch.int32),
                        _pinned(n, torch.int32), _pinned(n, torch.int32)]
    else:
        eng.prepare(case["edgefactor"], case["alpha"], case["beta"])
    return state


def _levels(eng, out):
    eng.check(eng.L.b200bfs_get_levels(eng.h, out.data_ptr()))


def run(state):
    case, eng = state["case"], state["eng"]
    kind, ef, alpha, beta = case["kind"], case["edgefactor"], case["alpha"], case["beta"]
    if kind == "noalloc":
        pred = state["pred"]
        depth = b200bfs.bfs_noalloc(state["row_ptr"].data_ptr(), state["col"].data_ptr(),
                                    pred.numel(), state["root"], pred.data_ptr(),
                                    torch.cuda.current_stream().cuda_stream)
        return {"depth": depth, "levels": pred >> 48}
    if kind == "batch":
        eng.run_batch(state["keys"], ef, alpha, beta)
        depth = eng.batch_root_levels()
        n = state["levels"].numel() // case["fetch"]
        for i in range(case["fetch"]):
            eng.batch_select(i * case["roots"] // case["fetch"])
            _levels(eng, state["levels"][i * n:(i + 1) * n])
        return {"depth": depth, "levels": state["levels"]}
    out = {}
    if kind == "first":
        _build(eng, state)
        eng.prepare(ef, alpha, beta)
        gi = eng.info()
        out["graph"] = [gi.scale, gi.num_global_edges, gi.num_global_verts, gi.tree_vertices]
        eng.check(eng.L.b200bfs_get_csr(eng.h, *[a.data_ptr() for a in state["csr"]]))
        out["csr"] = state["csr"]
    records, reached = [], []
    for root in state["keys"]:
        records.append(eng.run(root, ef, alpha, beta))
        reached.append(eng.run_stats().visited)
    out["records"], out["reached"] = np.stack(records), np.array(reached)
    if kind == "validate":
        out["errors"], out["edges"] = eng.validate(state["keys"][0])
    _levels(eng, state["levels"])
    out["levels"] = state["levels"]
    return out


def work(case):
    """Bytes that a pass cannot do without. Searches: the pred array written, one neighbour id per
    reached vertex (about half of a Kronecker graph's ids have an edge). Levels: read and written.
    Validation and construction: every input edge read once; construction: the CSR written and copied."""
    n = case["verts"] or 1 << case["scale"]
    m = case["edges"] or case["edgefactor"] * n
    search = 8 * n + 4 * (n // 2)
    levels = 8 * n + 4 * n
    kind = case["kind"]
    if kind == "noalloc":
        b = search + 8 * n
    elif kind == "batch":
        # a mask per reached vertex, written for its level and read for its neighbours
        b = 16 * (n // 2) + 4 * (n // 2) + case["fetch"] * levels
    else:
        b = case["roots"] * search + levels
        if kind == "validate":
            b += 8 * m + 8 * n
        if kind == "first":
            b += 8 * m + 2 * (8 * m + 16 * (n // 2))
    return {"bytes": b, "flops": 0}


def tolerance(case):
    return "exact"
