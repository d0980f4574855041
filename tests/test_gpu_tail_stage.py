"""SM-pair kernels on word counts that end in any part of a packed stage of
eight words: a trailing 256-sample stage without samples is neither unpacked
nor multiplied."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_r2_close
from qld_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["pair", "batch"])
@pytest.mark.parametrize("K", [1, 4, 5, 17, 24, 25, 26, 27, 28, 29, 32, 33, 36, 37, 41, 68])
def test_tail_stage_against_oracle(gpu_ctx, K, kernel):
    m, n, S = 530, 370, 64 * K - 5
    T, _ = synth.all_pairs_workload(m=m + n, n=S, seed=K)
    T = T.numpy().view(np.uint64).copy()
    bc = oracle.bitcounts(T)
    ld = K + (K & 1)
    # what lies past a row's words must not count
    D = torch.full((m + n, ld), -1, dtype=torch.int64, device="cuda")
    D[:, :K] = torch.from_numpy(T.view(np.int64)).cuda()
    dbc = torch.from_numpy(bc.view(np.int32).copy()).cuda()
    gpu_ctx.set_option(api.OPT_R2_MODE, api.R2_EXACT)
    gpu_ctx.set_option(api.OPT_SM_PAIR, 2 if kernel == "pair" else 0)
    r2 = torch.full((n, m), -3.0, device="cuda")
    counts = torch.zeros(n, m, dtype=torch.int32, device="cuda")
    args = dict(A=D[:m], bcA=dbc[:m], m=m, lda=ld, B=D[m:], bcB=dbc[m:], n=n, ldb=ld, K=K, S=S,
                symmetric=False, r2=r2, ldr=m, counts=counts, ldc=m)
    st = torch.cuda.current_stream()
    if kernel == "batch":
        gpu_ctx.ld_batch([args], stream=st)
    else:
        gpu_ctx.ld_device(stream=st, **args)
    gpu_ctx.sync(stream=st)
    want = oracle.counts(T[:m], T[m:])
    assert np.array_equal(counts.cpu().numpy().view(np.uint32), want)
    assert_r2_close(r2.cpu().numpy(), oracle.r2_exact(bc[:m], bc[m:], want, S))
