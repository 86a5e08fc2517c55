"""Many graphs in one launch: every configuration on batches whose packed
edge arrays start at any offset from a 16-byte boundary, with reached vertices
without out-edges, rows < cols, single vertices, empty edge lists and degrees
around a chunk, a warp round and a tile; clusters share graphs of any size
here (few graphs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def directed(B, rng, n, m, hub, less):
    src = rng.integers(0, n, m)
    dst = rng.integers(0, n, m)
    src = np.concatenate([src, np.zeros(hub, np.int64)])
    dst = np.concatenate([dst, rng.integers(0, n, hub)])
    order = np.argsort(src, kind="stable")
    indptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return B.Csc(indptr, dst[order], n - less, n)


@pytest.mark.parametrize("seed", [1, 2])
def test_every_configuration(B, O, seed):
    torch = torch_cuda()
    rng = np.random.default_rng(seed)
    shapes = [(1, 0, 0, 0), (2, 3, 1, 0), (33, 61, 4, 5), (700, 1403, 129, 100), (5000, 40001, 515, 0),
              (3001, 2999, 2050, 1), (40000, 300007, 9000, 777), (70000, 500003, 3, 0)]
    graphs = [directed(B, rng, *s) for s in shapes]
    roots = np.array([0 if i % 2 else rng.integers(0, g.n_cols) for i, g in enumerate(graphs)], np.uint32)
    refs = [O.oracle_bfs_queue(g.indptr, g.inds, int(r), g.n_rows, g.n_cols)
            for g, r in zip(graphs, roots)]
    batch = B.MultiBatch(graphs)
    out = torch.empty(batch.total_cols, dtype=torch.int32, device="cuda")
    for block, ipt, cluster in B.MULTI_CONFIGS_ALL:
        out.fill_(5)
        ec, _ = batch.run(roots, out.data_ptr(), block, ipt, cluster)
        lv = out.cpu().numpy()
        for i, (ref, edges) in enumerate(refs):
            o = batch.offset(i)
            assert np.array_equal(lv[o:o + len(ref)], ref), (block, ipt, cluster, i)
            assert ec[i] == edges, (block, ipt, cluster, i)
    batch.free()
