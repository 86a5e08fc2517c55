"""The hub layout is built by the first run whose plan reads it, not by runs of
fixed LLB and SLB plans."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("first", ["llb", "slb"])
@pytest.mark.parametrize("second", ["glb", "learned"])
def test_llb_and_slb_runs_take_no_memory_for_a_layout(B, O, first, second):
    """R-MAT 20: the layout is a copy of 31 M edges (125 MB), well above what a
    run may allocate besides (loop graphs and output scratch, 4 MB per array of
    vertices); levels, parents and edge counts before, through and after it."""
    torch = torch_cuda()
    dg = B.Graph.gen_rmat_device(20, 16, seed=7)
    layout_bytes = 4 * dg.nnz
    rng = np.random.default_rng(1)
    dg.sched_attach(rng.normal(0, 1.0, B.SCHED_PARAMS).astype(np.float32))
    g = dg.download()
    roots = [int(r) for r in B.sample_roots(g, 2, 7)]
    refs = [O.oracle_bfs_queue(g.indptr, g.inds, r) for r in roots]
    pinned = [torch.empty(g.n_cols, dtype=torch.int32, pin_memory=True) for _ in roots]

    def search(lb):
        for loop in ("graph", "host"):
            for r, (ref, ec) in zip(roots, refs):
                lv, pa, st = dg.run(r, B.options(lb, 256, loop=loop), parents=True)
                assert np.array_equal(lv, ref) and st.edges_count == ec, (lb, loop)
                kids = np.flatnonzero(ref > 0)
                assert np.all(ref[pa[kids]] == ref[kids] - 1) and pa[r] == r
        sts = dg.run_roots(roots, [t.data_ptr() for t in pinned], opts=B.options(lb, 256))
        for t, st, (ref, ec) in zip(pinned, sts, refs):
            assert np.array_equal(t.numpy(), ref) and st.edges_count == ec, lb

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    before = free()
    search(first)
    assert before - free() < layout_bytes // 2
    at = free()
    search(second)
    assert at - free() >= layout_bytes
    assert dg.hub_info()[1]
    search(first)
    dg.free()
