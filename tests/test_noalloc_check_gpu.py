"""bfs_run_device_noalloc on a malformed CSC: the check and the search's first
kernels are queued together, so the check has to leave the search without rows.
The call reports the graph, writes no level, and the next call is right."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("fault", ["nnz", "offsets", "target"])
@pytest.mark.parametrize("scale", [10, 15])
def test_malformed_csc_is_reported_and_searches_nothing(B, O, fault, scale):
    """Scale 10: every level is narrow; 15: wide ones too.  Every offset and
    index stays inside the arrays but the one target, which equals n_cols."""
    torch = torch_cuda()
    f = B.lib().bfs_run_device_noalloc
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint64, C.c_uint32,
                  C.c_void_p, C.POINTER(C.c_uint64), C.c_void_p]
    f.restype = C.c_int
    g = B.gen_rmat(scale, 16, seed=3)
    root = int(B.sample_roots(g, 1, 3)[0])
    ref, ec = O.oracle_bfs(g.indptr, g.inds, root)
    indptr, inds, nnz = g.indptr.copy(), g.inds.copy(), g.nnz
    if fault == "nnz":
        nnz -= 1
    elif fault == "offsets":
        v = int(np.flatnonzero((g.degree() > 0) & (np.arange(g.n_cols) != root))[3])
        indptr[v + 1] = indptr[v] - 1  # decreasing
    else:
        inds[int(g.indptr[root])] = g.n_cols

    def search(ip, ix, edges_in_array):
        ip = torch.from_numpy(ip.view(np.int32)).cuda()
        ix = torch.from_numpy(ix.view(np.int32)).cuda()
        out = torch.full((g.n_cols,), 7, dtype=torch.int32, device="cuda")
        edges = C.c_uint64(77)
        rc = f(ip.data_ptr(), ix.data_ptr(), g.n_rows, g.n_cols, edges_in_array, root, out.data_ptr(),
               C.byref(edges), None)
        torch.cuda.synchronize()
        return rc, out.cpu().numpy(), edges.value

    good = (g.indptr, g.inds, g.nnz)
    for _ in range(2):
        rc, out, edges = search(indptr, inds, nnz)
        assert B.STATUS[rc] == "BFS_ERR_GRAPH" and "malformed CSC" in B.lib().bfs_last_error().decode()
        assert np.all(out == 7) and edges == 77
        rc, out, edges = search(*good)
        assert rc == 0 and np.array_equal(out, ref) and edges == ec
