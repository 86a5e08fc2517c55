"""Lists ordered by target class and the edges to visited classes left out of
the frontier (csrc/hub_layout.cu, find_full_classes and level generation in
csrc/kernels.cu): list lengths around the limit between the two relabel
kernels, class limits around the vertex count, directed and symmetric graphs,
vertices whose every edge is left out, a level cut in the middle of a chunk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def skewed(B, n, m, long_lists, seed, symmetric):
    """m random edges whose targets favour low logical ids, long lists of the
    given lengths on the first vertices, a tail of 40 vertices in a path; ids
    shuffled."""
    rng = np.random.default_rng(seed)
    perm = rng.permutation(n)
    src = [rng.integers(0, n - 40, m)]
    dst = [(rng.random(m) ** 4 * (n - 40)).astype(np.int64)]
    for i, d in enumerate(long_lists):
        src.append(np.full(d, i))
        dst.append(rng.integers(0, n - 40, d))
    tail = np.arange(n - 41, n)
    src.append(tail[:-1])
    dst.append(tail[1:])
    src.append(np.array([5]))
    dst.append(np.array([n - 41]))
    src, dst = np.concatenate(src), np.concatenate(dst)
    if symmetric:
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    src, dst = perm[src], perm[dst]
    order = np.lexsort((rng.permutation(len(src)), src))  # lists in random order
    indptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return B.Csc(indptr, dst[order])


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("n,K", [(300, 128), (2047, 128), (2100, 256), (20011, 128), (70001, 4096)])
def test_levels_with_classes_left_out(B, O, n, K, symmetric):
    torch_cuda()
    g = skewed(B, n, 12 * n, [255, 256, 257, 4095, 8191, 8192, 8193, 9001], n + K, symmetric)
    dg = B.Graph.upload(g)
    dg.hub_configure(K, min_edges=1)
    # a layout where the K highest in-degrees hold a quarter of the edges
    indeg = np.sort(np.bincount(g.inds, minlength=n))[::-1]
    has = 4 * int(indeg[:K].sum()) >= g.nnz
    assert dg.hub_info()[:2] == ((K, True) if has else (0, False))
    rng = np.random.default_rng(3)
    dg.sched_attach(rng.normal(0, 1.0, B.SCHED_PARAMS).astype(np.float32))
    # record=1 takes every level through the two-kernel loop with whole
    # frontiers; without it classes are left out and small levels are fused
    for r in B.sample_roots(g, 4, n):
        ref, ec = O.oracle_bfs_queue(g.indptr, g.inds, int(r))
        for lb, loop, record in (("glb", "graph", 0), ("glb", "host", 0), ("learned", "graph", 0),
                                 ("learned", "host", 0), ("glb", "graph", 1)):
            for parents in (False, True):
                lv, pa, st = dg.run(int(r), B.options(lb, 256, loop=loop, record=record),
                                    parents=parents)
                assert np.array_equal(lv, ref), (lb, loop, record)
                assert st.edges_count == ec and st.reached == int((ref >= 0).sum())
                assert st.num_levels == int(ref.max()) + 1
                if parents:
                    kids = np.flatnonzero(ref > 0)
                    assert np.all(ref[pa[kids]] == ref[kids] - 1)
                if record:
                    tab = st.levels_table()
                    assert sum(tab["edges"]) == ec
    dg.free()


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("n,K", [(2047, 128), (20011, 128), (70001, 4096)])
def test_batches_with_classes_left_out(B, O, n, K, symmetric):
    """Batched runs: a class is left out once all roots of the pass (64, and 6
    in the last) have reached it; depths past the 16 levels of history."""
    torch = torch_cuda()
    g = skewed(B, n, 12 * n, [255, 257, 9001], n, symmetric)
    dg = B.Graph.upload(g)
    dg.hub_configure(K, min_edges=1)
    roots = B.sample_roots(g, 70, n)
    roots[3] = roots[9]
    ref, rec = O.oracle_bfs_many(g.indptr, g.inds, roots, queue_form=True)
    out = torch.full((len(roots), n), 7, dtype=torch.int32, device="cuda")
    for loop in ("graph", "host"):
        ec, _ = dg.run_batch(roots, out.data_ptr(), loop=loop)
        assert np.array_equal(out.cpu().numpy(), ref) and np.array_equal(ec, rec), loop
    dg.free()
