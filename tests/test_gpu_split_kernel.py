"""GPU parity of the split 4-bit kernel (ld_mxf4_split.cu), which the automatic
choice gives a task whose tiles all run at once: counts bit-exact, r^2 within
1e-6 of FP64 / bit-identical to the reference's arithmetic, and nothing
written outside the task, at the edges of its tiles, stages and word splits."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_r2_close
from qld_b200 import api, synth

pytestmark = pytest.mark.gpu

SHAPES = [
    # m, n (None: single region), samples, band
    (1, 1, 1, 0), (16, None, 64, 0), (17, 33, 513, 0),        # one tile; K = 9: two splits, uneven
    (129, 15, 2560, 0), (257, 241, 2049, 0),                  # past a half tile, past a 240 tile
    (64, None, 50000, 0), (300, 257, 20000, 0),               # four pairs per tile
    (731, 530, 5008, 0), (700, None, 10000, 0),
    (1500, 700, 16622, 0), (2048, None, 4096, 0),             # two pairs, one pair per tile
    (2500, None, 1000, 0), (18000, 40, 300, 0),               # near the one-wave limit
    (700, None, 900, 37), (1200, None, 3000, 300), (300, None, 20000, 299),
]


def _want(A, B, n, S, mode):
    bcA, bcB = oracle.bitcounts(A), oracle.bitcounts(B)
    c = oracle.counts(A, B)
    r2 = oracle.r2_exact(bcA, bcB, c, S) if mode == api.R2_EXACT else \
        oracle.r2_reference(bcA, bcB, c, S, fma_contract=False)
    return c, r2


@pytest.mark.parametrize("mode", [api.R2_EXACT, api.R2_REFERENCE], ids=["exact", "reference"])
@pytest.mark.parametrize("m,n,samples,band", SHAPES)
def test_split_kernel_equals_oracle(gpu_ctx, m, n, samples, band, mode):
    gpu_ctx.set_option(api.OPT_R2_MODE, mode)
    single = n is None
    rows = m if single else m + n
    t, _ = synth.all_pairs_workload(m=rows, n=samples, seed=rows + samples)
    T = t.numpy().view(np.uint64)
    A, B = T[:m], (T[:m] if single else T[m:])
    n = m if single else n
    K = T.shape[1]
    ld = K + (K & 1) + 2
    dev = torch.device("cuda", 0)
    D = torch.full((rows, ld), -1, dtype=torch.int64, device=dev)   # words past K are never read
    D[:, :K] = t.to(dev)
    bc = torch.from_numpy(oracle.bitcounts(T).view(np.int32).copy()).to(dev)
    width = band if band else m
    r2 = torch.full((n, width + 5), -3.0, device=dev)
    cnt = torch.full((n, width + 3), -3, dtype=torch.int32, device=dev)
    st = torch.cuda.current_stream()
    if band:
        gpu_ctx.ld_band_device(D, bc, m, ld, K, samples, band, r2, width + 5, counts=cnt,
                               ldc=width + 3, stream=st)
    else:
        gpu_ctx.ld_device(D[:m], bc[:m], m, ld, D[m:], bc[m:], n, ld, K, samples, single, r2,
                          width + 5, counts=cnt, ldc=width + 3, stream=st)
    gpu_ctx.sync(stream=st)
    want_c, want_r2 = _want(A, B, n, samples, mode)
    i, j = np.arange(n)[:, None], np.arange(width)[None, :]
    if band:                                   # column d of row i is the pair (i, i + 1 + d)
        valid = i + 1 + j < m
        at = np.minimum(i + 1 + j, m - 1)
        want_c, want_r2 = want_c[i, at], want_r2[i, at]
    else:
        valid = (j >= i) if single else np.ones((n, m), bool)
    got_r2, got_c = r2.cpu().numpy(), cnt.cpu().numpy()
    assert np.all(got_r2[:, width:] == -3.0) and np.all(got_c[:, width:] == -3)
    got_r2, got_c = got_r2[:, :width], got_c[:, :width]
    assert np.all(got_r2[~valid] == -3.0) and np.all(got_c[~valid] == -3)
    assert np.array_equal(got_c[valid].view(np.uint32), want_c[valid])
    if mode == api.R2_EXACT:
        assert_r2_close(got_r2, want_r2, mask=valid)
    else:
        assert np.array_equal(got_r2[valid].view(np.uint32),
                              want_r2[valid].astype(np.float32).view(np.uint32))


def test_split_kernel_equals_pair_kernel_on_streams(gpu_ctx):
    """The persistent kernel (two SMs per tile forced) gives the same bits, and
    calls on two streams do not disturb each other."""
    t, S = synth.all_pairs_workload(m=1100, n=7000, seed=9)
    K = t.shape[1]
    dev = torch.device("cuda", 0)
    D = torch.zeros(1100, K + (K & 1), dtype=torch.int64, device=dev)
    D[:, :K] = t.to(dev)
    bc = synth.popcount_rows(D).to(torch.int32)
    ld = D.shape[1]
    out = [torch.zeros(1100, 1100, device=dev) for _ in range(3)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(4):
        for o, s in zip(out, streams):
            gpu_ctx.ld_device(D, bc, 1100, ld, None, None, 1100, ld, K, S, True, o, 1100, stream=s)
    for s in streams:
        gpu_ctx.sync(stream=s)
    gpu_ctx.set_option(api.OPT_SM_PAIR, 2)
    gpu_ctx.ld_device(D, bc, 1100, ld, None, None, 1100, ld, K, S, True, out[2], 1100,
                      stream=streams[0])
    gpu_ctx.sync(stream=streams[0])
    assert torch.equal(out[0], out[2]) and torch.equal(out[1], out[2])
