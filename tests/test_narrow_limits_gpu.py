"""The narrow-level kernel (csrc/narrow.cu) at its own limits, taken from the
sources: levels of kNarrowEdges edges and one more or less, entries of
kNarrowHeavy edges, frontiers around the list's tile, the list's limit and the
queues' limit that arrive from a wide level, exits to a wide level with entries
in the list and in the queues, and a level of more new vertices than the queues
hold.  The number of launches shows which levels were wide, so a case that no
longer sits at its limit fails."""
import ctypes as C
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "bfs-gpu-sycl_gb300", "csrc")


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def constant(name):
    for f in ("kernels.h", "narrow.cu"):
        with open(os.path.join(CSRC, f)) as src:
            m = re.search(rf"constexpr uint32_t {name} = ([0-9u< ]+);", src.read())
        if m:
            return eval(m.group(1).replace("u", ""))  # digits and shifts only
    raise AssertionError(name)


EDGES = constant("kNarrowEdges")
HEAVY = constant("kNarrowHeavy")
HEAVY_BOUND = constant("kNarrowHeavyBound")
LIST = constant("kNarrowList")
ENTRIES = constant("kNarrowEntries")
TILE = constant("kNarrowTile")
QUEUES = 16 * constant("kNarrowQueue")


def spread(count, total, lo=1):
    """`count` degrees of at least lo that add up to `total`, as even as they go."""
    d = np.full(count, lo, np.int64)
    rest = total - d.sum()
    assert rest >= 0
    d += rest // count
    d[:rest % count] += 1
    return d


def layered(B, degrees, seed, last=1):
    """Layer k's vertices have the out-degrees degrees[k] (layer 0: the root) and
    edges to layer k + 1 only, all of whose vertices they reach; the last layer
    has `last` vertices without edges.  Ids and lists are shuffled."""
    rng = np.random.default_rng(seed)
    sizes = [len(d) for d in degrees] + [last]
    starts = np.concatenate([[0], np.cumsum(sizes)])
    n = int(starts[-1])
    src, dst = [], []
    for k, d in enumerate(degrees):
        e, m = int(d.sum()), sizes[k + 1]
        assert e >= m
        to = np.concatenate([np.arange(m), rng.integers(0, max(m, 1), e - m)])
        src.append(np.repeat(starts[k] + np.arange(sizes[k]), d))
        dst.append(starts[k + 1] + rng.permutation(to))
    perm = rng.permutation(n)
    src, dst = perm[np.concatenate(src)], perm[np.concatenate(dst)]
    order = np.argsort(src, kind="stable")
    indptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return B.Csc(indptr, dst[order]), int(perm[0])


def wide_levels(degrees):
    """Wide levels of a layered graph, by the rules of csrc/kernels.h."""
    wide, inside, first = 0, False, True
    for d in degrees:
        d = d[d > 0]
        F, EF = len(d), int(d.sum())
        if F == 0:
            break
        if inside and not first:  # the kernel knows which entries are heavy
            narrow = EF <= EDGES and int((d > HEAVY).sum()) <= LIST
        else:  # after the root or a wide level: a bound on the degrees
            heavy = EF - F + 1 > HEAVY_BOUND
            narrow = EF <= EDGES and F <= ENTRIES and (not heavy or F <= LIST)
        wide += 0 if narrow else 1
        inside, first = narrow, False
    return wide


def tail(n=5):
    return [np.array([1])] * n


def noalloc(B, torch, ip, ix_ptr, g, root):
    f = B.lib().bfs_run_device_noalloc
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint64, C.c_uint32,
                  C.c_void_p, C.POINTER(C.c_uint64), C.c_void_p]
    f.restype = C.c_int
    out = torch.full((g.n_cols,), 7, dtype=torch.int32, device="cuda")
    edges = C.c_uint64(0)
    assert f(ip.data_ptr(), ix_ptr, g.n_rows, g.n_cols, g.nnz, root, out.data_ptr(),
             C.byref(edges), None) == 0, B.lib().bfs_last_error()
    return out.cpu().numpy(), edges.value


def check(B, O, g, root, wide, seed, shifts=(0, 1, 3)):
    torch = torch_cuda()
    ref, ec = O.oracle_bfs_queue(g.indptr, g.inds, root, g.n_rows, g.n_cols)
    w = np.random.default_rng(seed).normal(0, 1.0, B.SCHED_PARAMS).astype(np.float32)
    ip = torch.from_numpy(g.indptr.view(np.int32)).cuda()
    kids = np.flatnonzero(ref > 0)
    key = np.sort(np.repeat(np.arange(g.n_cols, dtype=np.int64), g.degree()) * g.n_cols + g.inds)
    for shift in shifts:
        ix = torch.zeros(g.nnz + 8, dtype=torch.int32, device="cuda")
        ix[shift:shift + g.nnz] = torch.from_numpy(g.inds.view(np.int32)).cuda()
        ix_ptr = ix.data_ptr() + 4 * shift
        dg = B.Graph.wrap_device(ip.data_ptr(), ix_ptr, g.n_rows, g.n_cols, g.nnz)
        dg.sched_attach(w)
        dg.hub_configure(0)  # whole frontiers
        for lb in ("llb", "glb", "slb", "learned"):
            for parents in (False, True):
                lv, pa, st = dg.run(root, B.options(lb, 256), parents=parents)
                assert np.array_equal(lv, ref) and st.edges_count == ec, (lb, shift, parents)
                assert st.reached == int((ref >= 0).sum()) and st.num_levels == int(ref.max()) + 1
                if wide is not None:
                    assert st.launches == 3 + 3 * wide, (lb, st.launches, wide)
                if parents:
                    p = pa[kids].astype(np.int64)
                    assert np.all(ref[p] == ref[kids] - 1) and np.all(pa[ref < 0] == -1)
                    at = np.searchsorted(key, p * g.n_cols + kids)
                    assert np.array_equal(key[at], p * g.n_cols + kids)  # an edge of the graph
        dg.hub_configure(128, min_edges=1)
        for lb in ("glb", "learned"):
            lv, _, st = dg.run(root, B.options(lb, 256))
            assert np.array_equal(lv, ref) and st.edges_count == ec, (lb, shift)
        dg.free()
        lv, edges = noalloc(B, torch, ip, ix_ptr, g, root)
        assert np.array_equal(lv, ref) and edges == ec


@pytest.mark.parametrize("more", [-1, 0, 1])
@pytest.mark.parametrize("entries", [1, 1000, 30000])
def test_levels_of_the_most_edges(B, O, entries, more):
    """A level of kNarrowEdges edges (and one less, one more) on one entry, on
    1000 entries of more than kNarrowHeavy edges (the list) and on 30000 light
    ones (the queues), reached from the root; a wide one is left through levels
    that are narrow again."""
    degrees = [np.array([entries]), spread(entries, EDGES + more), spread(400, 900),
               spread(700, 700)] + tail()
    assert wide_levels(degrees) == (1 if more > 0 else 0)
    g, root = layered(B, degrees, entries + more)
    check(B, O, g, root, wide_levels(degrees), 1)


@pytest.mark.parametrize("more", [0, 1])
def test_root_of_the_most_edges(B, O, more):
    degrees = [np.array([EDGES + more]), spread(3000, 4000), spread(100, 130)] + tail()
    assert wide_levels(degrees) == more
    g, root = layered(B, degrees, more)
    check(B, O, g, root, more, 2, shifts=(0, 2))


@pytest.mark.parametrize("degree", [HEAVY - 1, HEAVY, HEAVY + 1])
def test_entries_at_the_heavy_limit(B, O, degree):
    degrees = [np.array([500]), np.full(500, degree), np.full(150, degree), spread(90, 100)] + tail()
    g, root = layered(B, degrees, degree)
    check(B, O, g, root, 0, 3)


# (entries, most edges of one): frontiers that a wide level leaves
ARRIVALS = [(n + k, heavy) for n in (TILE, LIST, ENTRIES) for k in (-1, 0, 1)
            for heavy in (0, HEAVY_BOUND + 100)]


@pytest.mark.parametrize("entries,heavy", ARRIVALS)
def test_frontiers_from_a_wide_level(B, O, entries, heavy):
    """The list takes frontiers with heavy entries up to kNarrowList entries, a
    tile of kNarrowTile at a time; light ones of more than a tile go into the
    queues, up to kNarrowEntries."""
    d = np.ones(entries, np.int64)
    d[entries // 3] += heavy
    d[:200] += 1
    degrees = [np.array([2500]), spread(2500, EDGES + 10), d, spread(300, 400)] + tail()
    wide = 1 + int(entries > (LIST if heavy else ENTRIES))
    assert wide_levels(degrees) == wide
    g, root = layered(B, degrees, entries + heavy)
    check(B, O, g, root, wide, 4, shifts=(0, 3))


@pytest.mark.parametrize("rows_less", [0, 5000])
def test_exit_with_list_and_queue_entries(B, O, rows_less):
    """The exit to a wide level puts the list's entries, then the blocks' queues,
    into one queue with its chunk prefix; twice, with narrow levels between."""
    mixed = np.concatenate([np.full(900, HEAVY + 30), np.full(22000, 3)])
    assert int(mixed.sum()) > EDGES
    degrees = [np.array([800]), spread(800, len(mixed)), mixed, spread(5000, 6000),
               spread(2000, len(mixed)), mixed, spread(50, 60)] + tail()
    assert wide_levels(degrees) == 2
    g, root = layered(B, degrees, 9)
    if rows_less:
        g = B.Csc(g.indptr, g.inds, g.n_cols - rows_less, g.n_cols)
    check(B, O, g, root, None if rows_less else 2, 5)


@pytest.mark.parametrize("over", [1500, 4000, 24000])
def test_more_new_vertices_than_the_queues_hold(B, O, over):
    """More new vertices with edges than the 16 queues' slots: the rest go to the
    list.  Whether the next level is wide depends on how the blocks' queues
    filled; with more than kNarrowList entries over it always is."""
    count = QUEUES + over
    assert count <= EDGES
    degrees = [np.array([2000]), spread(2000, count), np.ones(count, np.int64), spread(300, 500)] + tail()
    degrees[2][:5] += 2
    g, root = layered(B, degrees, over)
    if over > LIST:
        torch_cuda()
        dg = B.Graph.upload(g)
        assert dg.run(root, B.options("llb", 256))[2].launches == 3 + 3
        dg.free()
    check(B, O, g, root, None, 6)
