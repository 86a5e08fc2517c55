"""Levels of few edges run in one launch (csrc/narrow.cu), at the sizes where
its rules and tiles change: level sizes around the narrow limit, heavy entries
around the scan tile and the entry limit, single chunks, edges past the level
limit of the one-byte levels, rows < cols, misaligned edge arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def fan(B, mids, degs, n_leaves, tail, seed, n_rows_less=0):
    """Root -> `mids` vertices; mid i has degs[i] random leaves (duplicates and
    already reached vertices among them); leaf 0 starts a path of `tail`
    vertices.  Vertex ids are shuffled."""
    rng = np.random.default_rng(seed)
    n = 1 + mids + n_leaves + tail
    perm = rng.permutation(n)
    src = [np.zeros(mids, np.int64)]
    dst = [1 + np.arange(mids)]
    for i, d in enumerate(degs):
        src.append(np.full(d, 1 + i))
        dst.append(1 + mids + rng.integers(0, n_leaves, d))
    first = 1 + mids + n_leaves
    if tail:
        src.append(np.array([1]))
        dst.append(np.array([1 + mids]))
        chain = np.concatenate([[1 + mids], first + np.arange(tail)])
        src.append(chain[:-1])
        dst.append(chain[1:])
    src, dst = perm[np.concatenate(src)], perm[np.concatenate(dst)]
    order = np.argsort(src, kind="stable")
    indptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return B.Csc(indptr, dst[order], n - n_rows_less, n), int(perm[0])


def degrees(mids, total, heavy):
    """`mids` degrees >= 1 that add up to `total`, `heavy` of them on one."""
    d = np.ones(mids, np.int64)
    rest = total - mids
    d[mids // 2] += min(heavy, rest)
    rest -= min(heavy, rest)
    d += rest // mids
    d[:rest % mids] += 1
    return d


CASES = [(1, 1, 0), (1, 129, 0), (31, 70, 0), (33, 512, 300), (2047, 9000, 1000),
         (2048, 9000, 1000), (2049, 9000, 129), (8191, 60000, 2000), (8192, 60000, 2000),
         (8193, 60000, 2000), (700, 65535, 0), (700, 65536, 0), (700, 65537, 0),
         (16500, 65000, 0), (40000, 65536, 0)]


@pytest.mark.parametrize("mids,total,heavy", CASES)
def test_level_sizes_around_the_limits(B, O, mids, total, heavy):
    torch = torch_cuda()
    rng = np.random.default_rng(mids + total)
    weights = rng.normal(0, 1.0, B.SCHED_PARAMS).astype(np.float32)
    for shift in (0, 1, 3):
        g, root = fan(B, mids, degrees(mids, total, heavy), 50000, 300, 7 + shift)
        ref, ec = O.oracle_bfs_queue(g.indptr, g.inds, root)
        ip = torch.from_numpy(g.indptr.view(np.int32)).cuda()
        ix = torch.zeros(g.nnz + 8, dtype=torch.int32, device="cuda")
        ix[shift:shift + g.nnz] = torch.from_numpy(g.inds.view(np.int32)).cuda()
        dg = B.Graph.wrap_device(ip.data_ptr(), ix.data_ptr() + 4 * shift, g.n_rows, g.n_cols, g.nnz)
        dg.sched_attach(weights)
        for lb in ("llb", "glb", "slb", "learned"):
            for parents in (False, True):
                lv, pa, st = dg.run(root, B.options(lb, 256), parents=parents)
                assert np.array_equal(lv, ref) and st.edges_count == ec, (lb, shift)
                assert st.reached == int((ref >= 0).sum()) and st.num_levels == int(ref.max()) + 1
                if parents:
                    kids = np.flatnonzero(ref > 0)
                    assert np.all(ref[pa[kids]] == ref[kids] - 1) and np.all(pa[ref < 0] == -1)
                    edges = set(zip(np.repeat(np.arange(g.n_cols), g.degree()).tolist(),
                                    g.inds.tolist())) if total < 10000 else None
                    assert edges is None or all((int(pa[v]), int(v)) in edges for v in kids)
        dg.free()


def test_rows_lt_cols(B, O):
    torch_cuda()
    g, root = fan(B, 600, degrees(600, 30000, 400), 20000, 40, 3)
    for less in (1, 777, 9000):
        n_rows = g.n_cols - less
        ref, ec = O.oracle_bfs_queue(g.indptr, g.inds, root, n_rows, g.n_cols)
        dg = B.Graph.upload(B.Csc(g.indptr, g.inds, n_rows, g.n_cols))
        lv, _, st = dg.run(root, B.options("glb", 256))
        assert np.array_equal(lv, ref) and st.edges_count == ec
        dg.free()


def test_record_runs_every_level_in_its_arm(B):
    torch_cuda()
    g, root = fan(B, 600, degrees(600, 30000, 400), 20000, 40, 3)
    dg = B.Graph.upload(g)
    lv, _, st = dg.run(root, B.options("slb", 512, record=1))
    lv2, _, st2 = dg.run(root, B.options("slb", 512))
    tab = st.levels_table()
    assert set(a for a, f in zip(tab["arm"], tab["frontier"]) if f) == {8}
    assert np.array_equal(lv, lv2) and st.edges_count == st2.edges_count
    assert st2.launches < st.launches  # the narrow kernel replaces launches
    dg.free()
