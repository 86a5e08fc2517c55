"""Many graphs in one launch where edges point at vertices without out-edges: in
batches with many such edges those vertices are kept out of the queues
(kLeafShare in csrc/multigraph.cu).  Shares on both sides of the line, vertex
counts around a bitmap word, rows < cols (targets past the rows are not
expandable either), graphs whose every target is a leaf or none is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def graph(B, rng, n, leaves, degree, less=0):
    """`leaves` of the n vertices have no out-edges; n - less rows."""
    live = max(1, n - leaves)
    src = np.concatenate([np.arange(live), rng.integers(0, live, live * (degree - 1))])
    dst = rng.integers(0, n, len(src))
    perm = rng.permutation(n)
    src, dst = perm[src], perm[dst]
    order = np.argsort(src, kind="stable")
    indptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return B.Csc(indptr, dst[order], n - less, n), int(perm[0])


def share(graphs):
    """Edges that point at vertices that are not expandable, of all edges."""
    bad = sum(int(((g.degree()[g.inds] == 0) | (g.inds >= g.n_rows)).sum()) for g in graphs)
    return bad / sum(g.nnz for g in graphs)


@pytest.mark.parametrize("fraction", [0.0, 0.24, 0.26, 0.9])
def test_every_configuration(B, O, fraction):
    torch = torch_cuda()
    rng = np.random.default_rng(int(100 * fraction) + 1)
    sizes = [31, 32, 33, 63, 64, 65, 1, 700, 5000, 40000]
    made = [graph(B, rng, n, int(round(n * fraction)), 8) for n in sizes]
    graphs = [m[0] for m in made]
    assert (share(graphs) >= 0.25) == (fraction > 0.25)
    if fraction > 0.25:  # rows < cols, and a star, beside them
        made += [graph(B, rng, 3001, 700, 6, less) for less in (1, 33, 1500)]
        n = 2000
        made.append((B.Csc(np.concatenate([[0], np.full(n, n - 1)]), 1 + np.arange(n - 1)), 0))
        graphs = [m[0] for m in made]
        assert share(graphs) >= 0.25
    roots = [m[1] for m in made]
    refs = [O.oracle_bfs_queue(g.indptr, g.inds, r, g.n_rows, g.n_cols) for g, r in made]
    batch = B.MultiBatch(graphs)
    out = torch.empty(batch.total_cols, dtype=torch.int32, device="cuda")
    for cfg in B.MULTI_CONFIGS_ALL:
        out.fill_(5)
        ec, _ = batch.run(roots, out.data_ptr(), *cfg)
        lv = out.cpu().numpy()
        for i, (ref, edges) in enumerate(refs):
            o = batch.offset(i)
            assert np.array_equal(lv[o:o + len(ref)], ref) and ec[i] == edges, (cfg, i)
    batch.free()


def test_batch_without_edges(B):
    torch = torch_cuda()
    batch = B.MultiBatch([B.Csc(np.zeros(n + 1, np.uint32), np.zeros(0, np.uint32)) for n in (1, 40)])
    out = torch.full((41,), 5, dtype=torch.int32, device="cuda")
    ec, _ = batch.run([0, 7], out.data_ptr(), 256, 2, 1)
    want = np.full(41, -1)
    want[0] = want[1 + 7] = 0
    assert np.array_equal(out.cpu().numpy(), want) and list(ec) == [0, 0]
    batch.free()


def test_bitmap_larger_than_the_queues(B, O):
    """One row, 2^18 columns: the queues hold fewer words than the bitmap of
    expandable vertices, which then has memory of its own from the start."""
    torch = torch_cuda()
    rng = np.random.default_rng(4)
    n = 1 << 18
    indptr = np.full(n + 1, 6000, np.uint32)
    indptr[0] = 0
    graphs = [B.Csc(indptr, rng.integers(0, n, 6000), 1, n) for _ in range(2)]
    batch = B.MultiBatch(graphs)
    out = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    for roots in ([0, 0], [0, 77]):
        refs = [O.oracle_bfs_queue(g.indptr, g.inds, r, 1, n) for g, r in zip(graphs, roots)]
        for cfg in ((128, 1, 1), (512, 2, 1), (256, 4, 2), (512, 2, 8)):
            out.fill_(5)
            ec, _ = batch.run(roots, out.data_ptr(), *cfg)
            lv = out.cpu().numpy()
            for i, (ref, edges) in enumerate(refs):
                assert np.array_equal(lv[i * n:(i + 1) * n], ref) and ec[i] == edges, (cfg, i)
    batch.free()
