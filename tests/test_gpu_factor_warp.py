"""SM-pair kernel, column factors from a warp of their own or from the epilogue
warps: the choice goes by K (exact mode up to 100 words, reference mode up to
160) on launches of more than two waves of tiles.  A word of zeros appended to
every row changes neither the bit counts nor the pair counts, so the launch
just past the line must give the same bits as the one on it."""
import pytest
import torch

from qld_b200 import api, synth

pytestmark = pytest.mark.gpu


def _table(rows, K, S, seed):
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(seed)
    T = torch.randint(-2**63, 2**63 - 1, (rows, K), device=dev, dtype=torch.int64, generator=g)
    T[:, -1] &= (1 << (S - 64 * (K - 1))) - 1 if S < 64 * K else -1
    T[3] = 0                                           # an empty SNP and, once, a fixed one
    if seed % 2:
        T[rows - 5] = -1
        T[rows - 5, -1] = (1 << (S - 64 * (K - 1))) - 1
    return T


@pytest.mark.parametrize("kind,m,n,counts,seed", [
    ("region", 4993, 4993, False, 1), ("region", 5120, 5120, True, 2),
    ("pair", 4099, 4801, False, 3), ("pair", 4097, 4640, True, 4),
    ("band", 30011, 700, False, 5), ("band", 9001, 2403, False, 6)])
@pytest.mark.parametrize("mode,K", [("exact", 100), ("reference", 160)])
def test_factor_warp_against_epilogue_warps(gpu_ctx, kind, m, n, counts, seed, mode, K):
    dev, S = torch.device("cuda", 0), 64 * K - 13
    gpu_ctx.set_option(api.OPT_R2_MODE, api.R2_REFERENCE if mode == "reference" else api.R2_EXACT)
    T = _table(m + (n if kind == "pair" else 0), K, S, seed)
    ld = K + 2                                         # rows of whole 16 bytes
    t = torch.zeros((T.shape[0], ld), dtype=torch.int64, device=dev)
    t[:, :K] = T
    bc = synth.popcount_rows(t).to(torch.int32)
    got = []
    for words in (K, K + 1):
        st = torch.cuda.current_stream()
        if kind == "band":
            out, cnt = torch.full((m, n), -1.0, device=dev), None
            gpu_ctx.ld_band_device(t, bc, m, ld, words, S, n, out, n, stream=st)
        else:
            sym = kind == "region"
            out = torch.full((n, m), -1.0, device=dev)
            cnt = torch.full((n, m), -1, dtype=torch.int32, device=dev) if counts else None
            B = (None, None) if sym else (t[m:], bc[m:])
            gpu_ctx.ld_device(t[:m], bc[:m], m, ld, B[0], B[1], n, ld, words, S, sym, out, m,
                          counts=cnt, ldc=m if counts else 0, stream=st)
        gpu_ctx.sync(st)
        got.append((out, cnt))
    assert torch.equal(got[0][0].view(torch.int32), got[1][0].view(torch.int32))
    if counts:
        assert torch.equal(got[0][1], got[1][1])
    # and the line itself holds values, not the fill
    r = got[0][0]
    assert int((r >= 0).sum()) > r.numel() // 3
