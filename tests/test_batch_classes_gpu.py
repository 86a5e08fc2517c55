"""Batches look for target classes that every root has reached only on levels of
many edges (ms_looks in csrc/msbfs.cu); what is known stays known on the others.
Default thresholds, graphs whose levels lie on both sides of them, one root to a
full pass and more, searches that end with levels of few edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def with_tail(B, n, m, tail, seed):
    """m random symmetric edges with skewed targets among the first n - tail
    vertices, and a path of the other `tail` vertices that starts at vertex 5."""
    rng = np.random.default_rng(seed)
    body = n - tail
    src = rng.integers(0, body, m)
    dst = (rng.random(m) ** 4 * body).astype(np.int64)
    path = np.concatenate([[5], np.arange(body, n)])
    src, dst = np.concatenate([src, path[:-1]]), np.concatenate([dst, path[1:]])
    src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    perm = rng.permutation(n)
    src, dst = perm[src], perm[dst]
    order = np.argsort(src, kind="stable")
    indptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return B.Csc(indptr, dst[order])


@pytest.mark.parametrize("count", [1, 2, 5, 64, 70])
@pytest.mark.parametrize("n,K,average", [(70001, 4096, 12), (70001, 4096, 3), (300007, 16384, 6)])
def test_levels_on_both_sides_of_the_look(B, O, n, K, average, count):
    torch = torch_cuda()
    g = with_tail(B, n, average * n // 2, 30, n + average)
    dg = B.Graph.upload(g)
    dg.hub_configure(K)
    assert dg.hub_info()[:2] == (K, True)
    roots = B.sample_roots(g, count, 3)
    ref, rec = O.oracle_bfs_many(g.indptr, g.inds, roots, queue_form=True)
    degree = g.degree()
    edges = [int(sum(degree[lv == d].sum() for lv in ref[:64])) for d in range(int(ref.max()) + 1)]
    if average == 12 and count >= 5:  # the levels' edges, over the roots: both sides of 2^17
        assert max(edges) > 1 << 18 and min(edges) < 1000
    out = torch.full((count, n), 7, dtype=torch.int32, device="cuda")
    for loop in ("graph", "host"):
        ec, _ = dg.run_batch(roots, out.data_ptr(), loop=loop)
        assert np.array_equal(out.cpu().numpy(), ref) and np.array_equal(ec, rec), loop
    dg.free()
