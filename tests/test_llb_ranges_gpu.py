"""LLB's ranges (explore_local_body in csrc/kernels.cu): a level's 16-byte edge
chunks cut into equal ranges, one per block, none below the block size, entries
shared where a cut falls inside them.  Levels whose chunk count lies at the
edges of one range, of one range per block and of longer ranges; a long entry
over several ranges in front, in the middle and at the end; every alignment of
the edge array; the arm's own kernel and the one kernel for any arm.  Recorded
runs: every level then runs its arm's explore kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def chunks(first, degree, shift):
    return (first + shift + degree - 1) // 4 - (first + shift) // 4 + 1


def two_levels(B, target, where, shift, seed):
    """Vertex 0 -> mids 1 .. m -> leaves; the mids' edges make exactly `target`
    chunks, those over the random degrees' on the mid at `where` (0 .. 1)."""
    rng = np.random.default_rng(seed)
    m = max(1, min(700, target // 12))
    deg = rng.integers(1, 30, m)
    if m == 1:
        deg[:] = 1

    def total():
        first = m + np.concatenate([[0], np.cumsum(deg)[:-1]])  # after the root's list
        return int(sum(chunks(f, d, shift) for f, d in zip(first, deg)))

    at = int(where * (m - 1))
    deg[at] += 4 * (target - total())  # 4 edges more are one chunk more
    assert deg[at] > 0 and total() == target
    n_leaves = 4000
    n = 1 + m + n_leaves
    indptr = np.concatenate([[0], np.cumsum(np.concatenate([[m], deg, np.zeros(n_leaves, np.int64)]))])
    inds = np.concatenate([1 + np.arange(m), 1 + m + rng.integers(0, n_leaves, int(deg.sum()))])
    return B.Csc(indptr, inds)


def ranges_of(block, sms, ranges):
    return {"one": 1, "block-1": block - 1, "block": block, "block+1": block + 1,
            "grid-1": sms * block - 1, "grid": sms * block, "grid+1": sms * block + 1,
            "two": 2 * sms * block + 3}[ranges]


@pytest.mark.parametrize("ranges", ["one", "block-1", "block", "block+1", "grid-1", "grid", "grid+1",
                                    "two"])
@pytest.mark.parametrize("block", [128, 256, 512])
def test_levels_at_the_edges_of_the_ranges(B, O, block, ranges):
    torch = torch_cuda()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    target = ranges_of(block, sms, ranges)
    arm = {128: 0, 256: 1, 512: 2}[block]
    w = np.zeros(B.SCHED_PARAMS, np.float32)
    w[B.SCHED_PARAMS - B.SCHED_ARMS + arm] = 10.0  # the output bias: always this arm
    for shift, where in ((0, 0.5), (1, 1.0), (2, 0.0), (3, 0.7)):
        g = two_levels(B, target, where, shift, target + shift)
        ref, ec = O.oracle_bfs_queue(g.indptr, g.inds, 0)
        ip = torch.from_numpy(g.indptr.view(np.int32)).cuda()
        ix = torch.zeros(g.nnz + 8, dtype=torch.int32, device="cuda")
        ix[shift:shift + g.nnz] = torch.from_numpy(g.inds.view(np.int32)).cuda()
        dg = B.Graph.wrap_device(ip.data_ptr(), ix.data_ptr() + 4 * shift, g.n_rows, g.n_cols, g.nnz)
        dg.hub_configure(0)
        dg.sched_attach(w)
        edges = set((np.repeat(np.arange(g.n_cols), g.degree()) * g.n_cols + g.inds).tolist())
        for opts in (B.options("llb", block, sm_factor=1, record=1),
                     B.options("llb", block, record=1), B.options("llb", block, loop="host"),
                     B.options("learned", block, record=1)):
            for parents in (False, True):
                lv, pa, st = dg.run(0, opts, parents=parents)
                assert np.array_equal(lv, ref) and st.edges_count == ec
                if parents:
                    kids = np.flatnonzero(ref > 0)
                    assert all(int(pa[v]) * g.n_cols + int(v) in edges for v in kids)
                    assert np.all(ref[pa[kids]] == ref[kids] - 1) and np.all(pa[ref < 0] == -1)
                if opts.record:
                    assert st.levels_table()["arm"][1] == arm
        dg.free()
