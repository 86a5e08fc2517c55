"""What a batch of many graphs keeps between calls: the clusters' bitmaps after
an allocation that failed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HOOK = "BFS_GB300_FAIL_ALLOC_BYTES"


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def check(O, batch, graphs, roots, out, cfg):
    out.fill_(7)
    ec, _ = batch.run(roots, out.data_ptr(), *cfg)
    lv = out.cpu().numpy()
    for i, (g, r) in enumerate(zip(graphs, roots)):
        ref, edges = O.oracle_bfs_queue(g.indptr, g.inds, int(r), g.n_rows, g.n_cols)
        o = batch.offset(i)
        assert np.array_equal(lv[o:o + len(ref)], ref) and ec[i] == edges, (cfg, i)


def test_cluster_bitmaps_after_a_failed_allocation(B, O, monkeypatch):
    """Clusters of 2 need more bitmaps than clusters of 8 (2^18 vertices each,
    32 KiB: about 15 MB against 2.5); where they cannot be had the call reports
    it, and the next call with clusters of 8 has bitmaps of its own."""
    torch = torch_cuda()
    graphs = [B.gen_rmat(18, 4, seed=5), B.gen_rmat(10, 8, seed=6)]
    roots = [int(B.sample_roots(g, 1, 3)[0]) for g in graphs]
    batch = B.MultiBatch(graphs)
    out = torch.empty(batch.total_cols, dtype=torch.int32, device="cuda")
    check(O, batch, graphs, roots, out, (512, 2, 8))
    monkeypatch.setenv(HOOK, str(4 << 20))
    with pytest.raises(B.BfsError) as e:
        batch.run(roots, out.data_ptr(), 256, 2, 2)
    assert e.value.status == "BFS_ERR_OOM"
    check(O, batch, graphs, roots, out, (512, 2, 8))
    monkeypatch.delenv(HOOK)
    check(O, batch, graphs, roots, out, (256, 2, 2))
    batch.free()
