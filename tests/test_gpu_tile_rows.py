"""GPU parity of the SM-pair kernels' lower tiles: launches of a few waves, whose
tile height is chosen per launch, and batched tasks, whose tile rows share the
task's B rows evenly."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_r2_close
from qld_b200 import api, synth

pytestmark = pytest.mark.gpu
MODES = pytest.mark.parametrize("mode", [api.R2_EXACT, api.R2_REFERENCE],
                                ids=["exact", "reference"])


def _device_table(m, samples, seed):
    t, _ = synth.all_pairs_workload(m=m, n=samples, seed=seed)
    K = t.shape[1]
    D = torch.zeros(m, K + (K & 1), dtype=torch.int64, device="cuda")
    D[:, :K] = t.cuda()
    T = t.numpy().view(np.uint64)
    bc = oracle.bitcounts(T)
    return T, bc, D, torch.from_numpy(bc.view(np.int32).copy()).cuda(), K


def _check(got, counts, A, B, bcA, bcB, S, mode, mask):
    want = oracle.counts(A, B)
    if counts is not None:
        assert np.array_equal(counts.view(np.uint32)[mask], want[mask])
    if mode == api.R2_EXACT:
        assert_r2_close(got, oracle.r2_exact(bcA, bcB, want, S), mask=mask)
    else:
        ref = oracle.r2_reference(bcA, bcB, want, S, fma_contract=False)
        assert np.array_equal(got[mask].view(np.uint32), ref[mask].view(np.uint32))


@MODES
@pytest.mark.parametrize("m,n,samples", [(2700, None, 900), (3001, None, 5100),
                                         (2000, 3000, 300), (1537, 3601, 1000)])
def test_few_waves(gpu_ctx, m, n, samples, mode):
    gpu_ctx.set_option(api.OPT_R2_MODE, mode)
    single = n is None
    n = m if single else n
    T, bc, D, dbc, K = _device_table(m if single else m + n, samples, m + samples)
    A, B = T[:m], T[:m] if single else T[m:]
    bcB = bc[:m] if single else bc[m:]
    r2 = torch.full((n, m + 3), -3.0, device="cuda")
    cnt = torch.zeros(n, m, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream()
    gpu_ctx.ld_device(D[:m], dbc[:m], m, D.shape[1], D[m:], dbc[m:], n, D.shape[1], K, samples,
                      single, r2, m + 3, counts=cnt, ldc=m, stream=st)
    gpu_ctx.sync(stream=st)
    got = r2.cpu().numpy()
    mask = np.arange(m)[None, :] >= np.arange(n)[:, None] if single else np.ones((n, m), bool)
    assert np.all(got[:, m:] == -3.0) and np.all(got[:, :m][~mask] == -3.0)
    _check(got[:, :m], cnt.cpu().numpy(), A, B, bc[:m], bcB, samples, mode, mask)


@MODES
def test_batched_tile_heights(gpu_ctx, mode):
    gpu_ctx.set_option(api.OPT_R2_MODE, mode)
    T, bc, D, dbc, K = _device_table(900, 1500, 4)
    ld, S, jobs, tasks = D.shape[1], 1500, [], []
    for i, n in enumerate((1, 15, 16, 17, 128, 239, 240, 241, 250, 480, 481)):
        m = 1 + 61 * i % 400
        r2 = torch.full((n, m), -3.0, device="cuda")
        jobs.append(dict(A=D[:m], bcA=dbc[:m], m=m, lda=ld, B=D[400:], bcB=dbc[400:], n=n, ldb=ld,
                         K=K, S=S, symmetric=False, r2=r2, ldr=m))
        tasks.append((m, n, False, r2))
        r2s = torch.full((m, m), -3.0, device="cuda")
        jobs.append(dict(A=D[:m], bcA=dbc[:m], m=m, lda=ld, K=K, S=S, symmetric=True, r2=r2s,
                         ldr=m))
        tasks.append((m, m, True, r2s))
    st = torch.cuda.current_stream()
    gpu_ctx.ld_batch(jobs, stream=st)
    gpu_ctx.sync(stream=st)
    for m, n, single, r2 in tasks:
        got = r2.cpu().numpy()
        lo = 0 if single else 400
        mask = np.arange(m)[None, :] >= np.arange(n)[:, None] if single else np.ones((n, m), bool)
        assert np.all(got[~mask] == -3.0)
        _check(got, None, T[:m], T[lo:lo + n], bc[:m], bc[lo:lo + n], S, mode, mask)
