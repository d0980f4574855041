"""Counts beside exact r^2 on the SM-pair and split kernels: every entry a task
owes and no other, on tiles inside the task and across its edges and diagonal,
rows of any alignment."""
import numpy as np
import pytest
import torch

import oracle
from qld_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pair", [0, 2], ids=["auto", "pair"])
@pytest.mark.parametrize("m,n,pad", [(333, None, 0), (700, None, 1), (2900, None, 3),
                                     (257, 239, 7), (640, 480, 0), (769, 1001, 2),
                                     (3077, 2600, 1)])
def test_counts_of_the_window_only(gpu_ctx, m, n, pad, pair):
    S = 150
    single = n is None
    n = m if single else n
    t, _ = synth.all_pairs_workload(m=m if single else m + n, n=S, seed=m + pad)
    T = t.numpy().view(np.uint64)
    K = T.shape[1]
    D = torch.zeros(T.shape[0], K + (K & 1), dtype=torch.int64, device="cuda")
    D[:, :K] = t.cuda()
    bc = torch.from_numpy(oracle.bitcounts(T).view(np.int32).copy()).cuda()
    r2 = torch.full((n, m + pad), -3.0, device="cuda")
    cnt = torch.full((n, m + pad), -7, dtype=torch.int32, device="cuda")
    gpu_ctx.set_option(api.OPT_SM_PAIR, pair)
    st = torch.cuda.current_stream()
    gpu_ctx.ld_device(D[:m], bc[:m], m, D.shape[1], None if single else D[m:],
                      None if single else bc[m:], n, D.shape[1], K, S, single, r2, m + pad,
                      counts=cnt, ldc=m + pad, stream=st)
    gpu_ctx.sync(stream=st)
    keep = np.zeros((n, m + pad), bool)
    keep[:, :m] = np.arange(m)[None, :] >= np.arange(n)[:, None] if single else True
    got = cnt.cpu().numpy()
    want = oracle.counts(T[:m], T[:m] if single else T[m:])
    assert np.array_equal(got[keep], want.astype(np.int32)[keep[:, :m]])
    assert np.all(got[~keep] == -7) and np.all(r2.cpu().numpy()[~keep] == -3.0)
