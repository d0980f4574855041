"""The SM-pair kernel's tiles of fewer than 240 rows without counts, for two
regions, a single region and a band of a few waves, and its factor warp, against
the oracle; tables with empty and fixed SNPs, whose tiles fall back to the full
epilogue, and entries that must stay unwritten."""
import numpy as np
import pytest
import torch

import oracle
from conftest import assert_r2_close
from qld_b200 import api

pytestmark = pytest.mark.gpu
MODES = pytest.mark.parametrize("mode", [api.R2_EXACT, api.R2_REFERENCE],
                                ids=["exact", "reference"])


def _table(rows, S, rare, seed):
    """(host words, bit counts, device words, device bit counts) of random SNPs, one
    in eighteen empty and one in seventeen fixed if `rare`."""
    rng = np.random.default_rng(seed)
    K = (S + 63) // 64
    f = rng.integers(0, 1 << 64, (rows, K), dtype=np.uint64)
    T = np.where(rng.random((rows, 1)) < 0.5, f, f & rng.integers(0, 1 << 64, (rows, K),
                                                                  dtype=np.uint64))
    mask = np.full(K, ~np.uint64(0))
    if S % 64:
        mask[-1] = ~np.uint64(0) << np.uint64(64 - S % 64)
    if rare:
        T[3::18] = 0
        T[5::17] = ~np.uint64(0)
    T &= mask
    bc = oracle.bitcounts(T)
    D = torch.zeros(rows, K + (K & 1), dtype=torch.int64, device="cuda")
    D[:, :K] = torch.from_numpy(T.view(np.int64)).cuda()
    return T, bc, D, torch.from_numpy(bc.view(np.int32).copy()).cuda()


def _check(got, A, bcA, B, bcB, S, mode, mask):
    want = oracle.counts(A, B)
    if mode == api.R2_EXACT:
        assert_r2_close(got, oracle.r2_exact(bcA, bcB, want, S), mask=mask)
    else:
        ref = oracle.r2_reference(bcA, bcB, want, S, fma_contract=False)
        assert np.array_equal(got.view(np.uint32)[mask], ref.view(np.uint32)[mask])


@MODES
@pytest.mark.parametrize("rare", [False, True], ids=["", "rare"])
@pytest.mark.parametrize("m,n,S", [(3001, None, 300), (2700, None, 1100), (2000, 3000, 257),
                                   (1537, 3601, 640)])
def test_regions(gpu_ctx, m, n, S, rare, mode):
    gpu_ctx.set_option(api.OPT_R2_MODE, mode)
    single = n is None
    n = m if single else n
    T, bc, D, dbc = _table(m if single else m + n, S, rare, m + S)
    out = torch.full((n, m + 3), -3.0, device="cuda")
    st = torch.cuda.current_stream()
    gpu_ctx.ld_device(D[:m], dbc[:m], m, D.shape[1], None if single else D[m:],
                      None if single else dbc[m:], n, D.shape[1], T.shape[1], S, single, out, m + 3,
                      stream=st)
    gpu_ctx.sync(stream=st)
    got = out.cpu().numpy()
    owed = np.arange(m)[None, :] >= np.arange(n)[:, None] if single else np.ones((n, m), bool)
    assert np.all(got[:, m:] == -3.0) and np.all(got[:, :m][~owed] == -3.0)
    b = 0 if single else m
    _check(np.ascontiguousarray(got[:, :m]), T[:m], bc[:m], T[b:b + n], bc[b:b + n], S, mode, owed)


@MODES
@pytest.mark.parametrize("rare", [False, True], ids=["", "rare"])
@pytest.mark.parametrize("m,W,S", [(4000, 1500, 300), (6001, 901, 700), (8001, 400, 270),
                                   (30011, 700, 6400)])
def test_bands(gpu_ctx, m, W, S, rare, mode):
    gpu_ctx.set_option(api.OPT_R2_MODE, mode)
    T, bc, D, dbc = _table(m, S, rare, W)
    out = torch.full((m, W), -3.0, device="cuda")
    st = torch.cuda.current_stream()
    gpu_ctx.ld_band_device(D, dbc, m, D.shape[1], T.shape[1], S, W, out, W, stream=st)
    gpu_ctx.sync(stream=st)
    got = out.cpu().numpy()
    past = np.arange(m)[:, None] + 1 + np.arange(W)[None, :] >= m
    assert np.all(got[past] == -3.0)
    rng = np.random.default_rng(W)
    for b in sorted({0, 3, 5, m - 2, m - W - 1, m - W, *map(int, rng.integers(0, m - 1, 40))}):
        a1 = min(m, b + 1 + W)
        row = got[b:b + 1, :a1 - b - 1]
        _check(np.ascontiguousarray(row), T[b + 1:a1], bc[b + 1:a1], T[b:b + 1], bc[b:b + 1], S, mode,
               np.ones(row.shape, bool))


# K at and past the lines of the factor warp's rule, more than two waves of tiles
@MODES
@pytest.mark.parametrize("K", [30, 100, 101, 160, 161])
@pytest.mark.parametrize("m,n", [(5009, None), (4100, 4700)])
def test_sampled_rows_of_many_waves(gpu_ctx, m, n, K, mode):
    gpu_ctx.set_option(api.OPT_R2_MODE, mode)
    single, S = n is None, 64 * K - 29
    n = m if single else n
    T, bc, D, dbc = _table(m if single else m + n, S, True, K)
    out = torch.full((n, m), -3.0, device="cuda")
    st = torch.cuda.current_stream()
    gpu_ctx.ld_device(D[:m], dbc[:m], m, D.shape[1], None if single else D[m:],
                      None if single else dbc[m:], n, D.shape[1], K, S, single, out, m, stream=st)
    gpu_ctx.sync(stream=st)
    rng = np.random.default_rng(K)
    at = 0 if single else m
    for b in sorted({0, 3, 5, n - 1, *map(int, rng.integers(0, n, 24))}):
        row = out[b:b + 1].cpu().numpy()
        owed = np.arange(m)[None, :] >= (b if single else 0)
        assert np.all(row[~owed] == -3.0)
        _check(row, T[:m], bc[:m], T[at + b:at + b + 1], bc[at + b:at + b + 1], S, mode, owed)
