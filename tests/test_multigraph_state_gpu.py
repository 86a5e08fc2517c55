"""What a batch of many graphs keeps between calls: the clusters' bitmaps after
an allocation that failed, and the file of tuned configurations; each kernel is
timed once."""
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


def uniform(B, n, m, seed):
    rng = np.random.default_rng(seed)
    src = np.sort(rng.integers(0, n, m))
    indptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return B.Csc(indptr, rng.integers(0, n, m))


@pytest.mark.parametrize("clusters", [False, True])
def test_tuned_configuration_is_reused_only_for_its_kernels_and_sizes(B, tmp_path, clusters):
    torch = torch_cuda()
    path = tmp_path / "tuned.tsv"

    def tune(graphs):
        batch = B.MultiBatch(graphs)
        out = torch.empty(batch.total_cols, dtype=torch.int32, device="cuda")
        best, times = batch.autotune([0] * len(graphs), out.data_ptr(), reps=1,
                                     cache_path=str(path), clusters=clusters)
        batch.free()
        return best, all(t > 0 for t in times)

    even = [uniform(B, 2000, 8000, 1), uniform(B, 2000, 8000, 2)]
    best, timed = tune(even)
    assert timed
    assert tune(even) == (best, False)  # from the file
    # equal numbers of graphs, vertices and edges, other sizes
    uneven = [uniform(B, 1000, 4000, 3), uniform(B, 3000, 12000, 4)]
    assert tune(uneven)[1]
    assert not tune(uneven)[1] and not tune(even)[1]
    # lines of another revision of the kernels, and of the key without one
    key, cfg = path.read_text().splitlines()[0].split("\t")
    head, sep, rev = key.rpartition("|r")
    assert sep
    path.write_text(f"{head}|r{int(rev) + 1}\t{cfg}\n{head}\t{cfg}\n{head.split('|h')[0]}\t{cfg}\n")
    assert tune(even)[1]


def test_each_kernel_is_timed_once(B):
    """Items per thread 2 and 4 name the same kernel: one time for both, and the
    choice is not left to noise between them."""
    torch = torch_cuda()
    batch = B.MultiBatch([uniform(B, 3000, 20000, s) for s in range(3)])
    out = torch.empty(batch.total_cols, dtype=torch.int32, device="cuda")
    for clusters in (False, True):
        best, times = batch.autotune([0, 1, 2], out.data_ptr(), reps=3, clusters=clusters)
        configs = B.MULTI_CONFIGS_ALL[:len(times)]
        t = dict(zip(configs, times))
        assert all(x > 0 for x in times)
        assert all(t[b, 2, c] == t[b, 4, c] for b, p, c in configs if p == 4)
        assert best[1] != 4 and t[(best + (1,))[:3]] == min(times)
    batch.free()
