"""GLB's walk of 16-byte edge chunks (explore_chunk_body in csrc/kernels.cu):
entries of every length around a round of 32 chunks, which takes the path for
rounds inside one entry, and levels at the chunk counts from which a lane walks
two chunks per group and from which claims are made together."""
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       "bfs-gpu-sycl_gb300", "csrc", "kernels.cu")


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def constant(name):
    with open(KERNELS) as src:
        m = re.search(rf"constexpr uint32_t {name} = ([0-9u< ]+);", src.read())
    return eval(m.group(1).replace("u", ""))  # digits and shifts only


@pytest.mark.parametrize("hub", [0, 128])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_entries_around_a_round_of_chunks(B, O, shift, hub):
    """Recorded runs, so that the level is not taken by the narrow kernel."""
    torch = torch_cuda()
    rng = np.random.default_rng(shift)
    deg = np.concatenate([np.arange(1, 13), np.arange(120, 137), np.arange(250, 263),
                          np.arange(380, 390), np.arange(505, 520), np.arange(1020, 1030), [4999]])
    deg = rng.permutation(np.repeat(deg, 5))
    m, n_leaves = len(deg), 6000
    n = 1 + m + n_leaves
    to = (rng.random(int(deg.sum())) ** 3 * n_leaves).astype(np.int64)  # low leaves are hubs
    indptr = np.concatenate([[0], np.cumsum(np.concatenate([[m], deg, np.zeros(n_leaves, np.int64)]))])
    g = B.Csc(indptr, np.concatenate([1 + np.arange(m), 1 + m + to]))
    ref, ec = O.oracle_bfs_queue(g.indptr, g.inds, 0)
    ip = torch.from_numpy(g.indptr.view(np.int32)).cuda()
    ix = torch.zeros(g.nnz + 8, dtype=torch.int32, device="cuda")
    ix[shift:shift + g.nnz] = torch.from_numpy(g.inds.view(np.int32)).cuda()
    dg = B.Graph.wrap_device(ip.data_ptr(), ix.data_ptr() + 4 * shift, n, n, g.nnz)
    dg.hub_configure(hub, min_edges=1)
    assert dg.hub_info()[:2] == ((hub, True) if hub else (0, False))
    lv = torch.empty(n, dtype=torch.int32, device="cuda")
    pa = torch.empty(n, dtype=torch.int32, device="cuda")
    for loop in ("graph", "host"):
        for ipt in (4, 8):
            opts = B.options("glb", 256, loop=loop, record=1, ipt=ipt)
            for parents in (None, pa.data_ptr()):
                st = dg.run_device(0, lv.data_ptr(), parents, opts)
                assert np.array_equal(lv.cpu().numpy(), ref) and st.edges_count == ec
            assert dg.validate_device(0, lv.data_ptr(), pa.data_ptr()) == 0
    dg.free()


@pytest.mark.parametrize("limit", ["kGroupChunks", "kPackedChunks"])
@pytest.mark.parametrize("more", [-1, 0])
def test_levels_around_the_chunk_limits(B, limit, more):
    """Vertex 0 -> mids -> leaves -> a path; the mids' edges make exactly the
    limit's number of chunks or one less.  A leaf's level is 2 exactly when some
    edge points at it.  Without a layout, and with one (whose own chunk count is
    near the limit): targets favour few leaves, and the filter is loaded."""
    torch = torch_cuda()
    target = constant(limit) + more
    gen = torch.Generator(device="cuda").manual_seed(5)
    m, n_leaves, path = 300000, 400000, 20
    average = 4 * target // m
    deg = torch.randint(1, 2 * average - 40, (m,), generator=gen, device="cuda")
    deg[7::997] = 3 * average

    def chunks():
        first = m + torch.cumsum(deg, 0) - deg  # after the root's list
        return int(((first + deg - 1) // 4 - first // 4 + 1).sum())

    deg[m // 2] += 4 * (target - chunks())
    assert int(deg[m // 2]) > 0 and chunks() == target
    total = int(deg.sum())
    at = torch.rand(total, generator=gen, device="cuda")
    to = (at * at * at * (n_leaves - 1)).to(torch.int32)
    del at
    hit = torch.zeros(n_leaves, dtype=torch.bool, device="cuda")
    hit[to.long()] = True
    hit[0] = True
    to[0] = 0  # leaf 0 starts the path
    first_leaf, n = 1 + m, 1 + m + n_leaves + path
    first_path = first_leaf + n_leaves
    to += first_leaf
    chain = torch.arange(first_path, n, dtype=torch.int32, device="cuda")
    inds = torch.cat([torch.arange(1, m + 1, dtype=torch.int32, device="cuda"), to, chain])
    degrees = torch.zeros(n, dtype=torch.int64, device="cuda")
    degrees[0], degrees[1:m + 1], degrees[first_leaf] = m, deg, 1
    degrees[first_path:n - 1] = 1
    indptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(degrees, 0, out=indptr[1:])
    indptr = indptr.to(torch.int32)
    assert int(indptr[-1]) == inds.numel()
    want = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    want[0], want[1:m + 1] = 0, 1
    want[first_leaf:first_path] = torch.where(hit, 2, -1).to(torch.int32)
    want[first_path:] = 3 + torch.arange(path, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    dg = B.Graph.wrap_device(indptr.data_ptr(), inds.data_ptr(), n, n, inds.numel())
    lv = torch.empty(n, dtype=torch.int32, device="cuda")
    pa = torch.empty(n, dtype=torch.int32, device="cuda")
    # a layout where the prefix's targets take a quarter of the edges: the larger
    # one's do, the smaller one's 22 %
    by_degree = torch.sort(torch.bincount(inds.long(), minlength=n), descending=True)[0]
    for hub in (0, 4096, 16384):
        dg.hub_configure(hub)
        has = 4 * int(by_degree[:hub].sum()) >= inds.numel()
        assert has == (hub == 16384)
        assert dg.hub_info()[:2] == ((hub, True) if has else (0, False))
        for loop in ("graph", "host"):
            for parents in (None, pa.data_ptr()):
                lv.fill_(7)
                st = dg.run_device(0, lv.data_ptr(), parents, B.options("glb", 256, loop=loop))
                assert torch.equal(lv, want), (hub, loop, parents)
                assert st.edges_count == inds.numel()
            assert dg.validate_device(0, lv.data_ptr(), pa.data_ptr()) == 0
    dg.free()
