"""Tables in which many SNPs are fixed (every sample carries the allele) or
empty: every pair of them against the oracle, on each kernel's epilogue, with
and without counts, in both r^2 modes."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_r2_close
from qld_b200 import api

pytestmark = pytest.mark.gpu


def _table(m, S, fixed, empty, seed):
    rng = np.random.default_rng(seed)
    bits = rng.random((m, S)) < rng.uniform(0.02, 0.98, (m, 1))
    kind = rng.random(m)
    bits[kind < fixed] = True
    bits[kind > 1 - empty] = False
    K = (S + 63) // 64
    padded = np.zeros((m, K * 64), bool)
    padded[:, :S] = bits
    return np.packbits(padded, axis=1).view(">u8").astype(np.uint64)


@pytest.mark.parametrize("kernel", ["split", "pair", "single", "batch", "mma", "popc"])
@pytest.mark.parametrize("mode", [api.R2_EXACT, api.R2_REFERENCE], ids=["exact", "reference"])
@pytest.mark.parametrize("S,fixed,empty", [(300, 0.2, 0.2), (1000, 0.05, 0.05), (257, 0.3, 0.0),
                                           (600, 0.0, 0.3), (70, 0.1, 0.1)])
def test_fixed_and_empty(gpu_ctx, S, fixed, empty, mode, kernel):
    m, n = (300, 290) if kernel == "split" else (530, 1500) if kernel == "pair" else (270, 500)
    T = _table(m + n, S, fixed, empty, S)
    bc = oracle.bitcounts(T)
    K, ld = T.shape[1], T.shape[1] + (T.shape[1] & 1)
    D = torch.zeros(m + n, ld, dtype=torch.int64, device="cuda")
    D[:, :K] = torch.from_numpy(T.view(np.int64)).cuda()
    dbc = torch.from_numpy(bc.view(np.int32).copy()).cuda()
    gpu_ctx.set_option(api.OPT_R2_MODE, mode)
    gpu_ctx.set_option(api.OPT_KERNEL, {"mma": api.KERNEL_MMA, "popc": api.KERNEL_POPC}.get(kernel, 0))
    gpu_ctx.set_option(api.OPT_SM_PAIR, {"pair": 2, "single": 1}.get(kernel, 0))
    st = torch.cuda.current_stream()
    want = oracle.counts(T[:m], T[m:])
    if mode == api.R2_EXACT:
        r2 = oracle.r2_exact(bc[:m], bc[m:], want, S)
    else:
        r2 = oracle.r2_reference(bc[:m], bc[m:], want, S, fma_contract=False)
    for counts in (None, torch.zeros(n, m, dtype=torch.int32, device="cuda")):
        out = torch.full((n, m), -3.0, device="cuda")
        args = dict(A=D[:m], bcA=dbc[:m], m=m, lda=ld, B=D[m:], bcB=dbc[m:], n=n, ldb=ld, K=K,
                    S=S, symmetric=False, r2=out, ldr=m, counts=counts,
                    ldc=0 if counts is None else m)
        if kernel == "batch":
            gpu_ctx.ld_batch([args], stream=st)
        else:
            gpu_ctx.ld_device(stream=st, **args)
        gpu_ctx.sync(stream=st)
        got = out.cpu().numpy()
        if mode == api.R2_EXACT:
            assert_r2_close(got, r2)
        else:
            assert np.array_equal(got.view(np.uint32), r2.view(np.uint32))
        if counts is not None:
            assert np.array_equal(counts.cpu().numpy(), want.astype(np.int32))
