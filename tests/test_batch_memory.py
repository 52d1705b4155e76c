"""An autotuned batch where the tensor-core filter runs on a sample but has no room for the class's largest set: the
tree answers it.  (Device memory is taken up to what the sample needs; nothing else allocates meanwhile.)"""

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")


@pytest.mark.parametrize("structure,n", [("ball", 3000), ("kd", 3000), ("ball", 60000)])
def test_filter_without_room_for_the_whole_set(structure, n):
    import torch
    from cudaexactknn_gb300 import knn
    rng = np.random.default_rng(n)
    pts, basis = W.subspace(rng, n, 16, 4, 0.05)
    qs, _ = W.subspace(rng, 250000, 16, 4, 0.05, basis)
    rows = np.arange(0, len(qs), 1000)
    want = oracle.bf_knn(pts, qs[rows], 5, fma=True, threads=8)
    ix = gu.make_index(structure, pts)
    dq = gu.to_dev(qs)
    gu.run(ix, qs[:100], 5)  # the kernels' own memory
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    # The filter keeps 1,024 candidates of 8 bytes per query: 2 GB for the set, 67 MB for the sample.
    taken = torch.empty(max(0, free - (1 << 30)), dtype=torch.uint8, device="cuda")
    try:
        batch = knn.Batch([(ix, dq, 5, float("inf"))], autotune=True)
        (idx, dist), = batch.run()
        got = idx.cpu().numpy()[rows], dist.cpu().numpy()[rows]
        batch.close()
    finally:
        del taken
        torch.cuda.empty_cache()
    gu.assert_rows_equal(*got, *want)
    ix.close()
