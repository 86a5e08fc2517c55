"""bfs_run_roots over more roots than it queues at a time (kRunsAhead in
csrc/engine.cu): a full window, one root past it, and a third window; results,
statistics and the two device slots across the windows' ends, for pinned and
pageable buffers, with and without parents, for plans that are queued ahead and
plans that the host drives."""
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ENGINE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "bfs-gpu-sycl_gb300", "csrc", "engine.cu")


def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def ahead():
    with open(ENGINE) as src:
        return int(re.search(r"constexpr uint32_t kRunsAhead = (\d+);", src.read()).group(1))


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("extra", [0, 1, 33])
def test_windows_of_roots(B, O, extra, pinned):
    torch = torch_cuda()
    g = B.gen_rmat(11, 8, seed=17)
    n, count = g.n_cols, ahead() + extra
    roots = [int(r) for r in B.sample_roots(g, min(count, 40), 17)]
    roots = (roots + roots[::-1])[:count]
    refs = {r: O.oracle_bfs(g.indptr, g.inds, r) for r in set(roots)}
    dg = B.Graph.upload(g)
    w = np.random.default_rng(17).normal(0, 1.0, B.SCHED_PARAMS).astype(np.float32)
    dg.sched_attach(w)
    lv = [torch.empty(n, dtype=torch.int32, pin_memory=pinned) for _ in roots]
    pa = [torch.empty(n, dtype=torch.int32, pin_memory=pinned) for _ in roots]
    for opts in (B.options("llb", 256), B.options("learned"), B.options("glb", 256, loop="host"),
                 B.options("glb", 256, record=1)):
        for parents in (False, True):
            for t in lv + pa:
                t.fill_(7)
            sts = dg.run_roots(roots, [t.data_ptr() for t in lv],
                               [t.data_ptr() for t in pa] if parents else None, opts)
            assert len(sts) == count
            for r, st, l, p in zip(roots, sts, lv, pa):
                ref, ec = refs[r]
                assert np.array_equal(l.numpy(), ref) and st.edges_count == ec
                assert st.reached == int((ref >= 0).sum()) and st.num_levels == int(ref.max()) + 1
                assert st.device_ms > 0 and st.launches >= 3
                assert (st.recorded > 0) == (opts.record > 0)
                pp = p.numpy()
                if parents:
                    kids = np.flatnonzero(ref > 0)
                    assert np.all(ref[pp[kids]] == ref[kids] - 1) and pp[r] == r
                else:
                    assert np.all(pp == 7)
    dg.free()
