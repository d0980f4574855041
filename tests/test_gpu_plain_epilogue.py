"""The SM-pair kernels' epilogue without counts against the one with counts and
against the oracle, on the rows it hands to the full form: empty and fixed
SNPs, bit counts that do not match the data (r^2 above 1.0001, counts above S),
few samples."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_r2_close
from qld_b200 import api, synth

pytestmark = pytest.mark.gpu


def _table(m, samples, rare, seed):
    t, _ = synth.all_pairs_workload(m=m, n=samples, seed=seed)
    T = t.numpy().view(np.uint64).copy()
    full = np.zeros(T.shape[1], np.uint64)
    for s in range(samples):
        full[s // 64] |= np.uint64(1) << np.uint64(63 - s % 64)
    if "fixed" in rare:
        T[3::97] = full
    if "empty" in rare:
        T[5::89] = 0
    bc = oracle.bitcounts(T)
    if "mismatch" in rare:                   # too small: r^2 > 1.0001; too large: above S
        bc[7::101] = np.maximum(bc[7::101] // 3, 1)
        bc[11::103] = samples + 7
    return T, bc


@pytest.mark.parametrize("kernel", ["split", "pair", "batch"])
@pytest.mark.parametrize("mode", [api.R2_EXACT, api.R2_REFERENCE], ids=["exact", "reference"])
@pytest.mark.parametrize("samples,rare", [(1500, ""), (1500, "fixed"), (1500, "empty"),
                                          (1500, "fixed empty"), (1500, "mismatch"),
                                          (700, "fixed empty mismatch"), (90, ""),
                                          (256, "fixed"), (255, "empty")])
def test_plain_equals_full(gpu_ctx, samples, rare, mode, kernel):
    m, n = (300, 290) if kernel == "split" else (700, 650)
    T, bc = _table(m + n, samples, rare.split(), samples + len(rare))
    K = T.shape[1]
    ld = K + (K & 1)
    D = torch.zeros(m + n, ld, dtype=torch.int64, device="cuda")
    D[:, :K] = torch.from_numpy(T.view(np.int64)).cuda()
    dbc = torch.from_numpy(bc.view(np.int32).copy()).cuda()
    gpu_ctx.set_option(api.OPT_R2_MODE, mode)
    gpu_ctx.set_option(api.OPT_SM_PAIR, 2 if kernel == "pair" else 0)
    st = torch.cuda.current_stream()
    out = []
    for counts in (None, torch.zeros(n, m, dtype=torch.int32, device="cuda")):
        r2 = torch.full((n, m), -3.0, device="cuda")
        args = dict(A=D[:m], bcA=dbc[:m], m=m, lda=ld, B=D[m:], bcB=dbc[m:], n=n, ldb=ld, K=K,
                    S=samples, symmetric=False, r2=r2, ldr=m, counts=counts,
                    ldc=0 if counts is None else m)
        if kernel == "batch":
            gpu_ctx.ld_batch([args], stream=st)
        else:
            gpu_ctx.ld_device(stream=st, **args)
        gpu_ctx.sync(stream=st)
        out.append(r2.cpu().numpy())
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
    want = oracle.counts(T[:m], T[m:])
    if mode == api.R2_EXACT:
        if "mismatch" not in rare:           # there the rule's side of 1.0001 may differ in FP32
            assert_r2_close(out[0], oracle.r2_exact(bc[:m], bc[m:], want, samples))
    else:
        ref = oracle.r2_reference(bc[:m], bc[m:], want, samples, fma_contract=False)
        same = out[0].view(np.uint32) == ref.view(np.uint32)
        assert np.all(same | (np.isnan(out[0]) & np.isnan(ref)))
