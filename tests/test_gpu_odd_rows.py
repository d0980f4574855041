"""Counts beside r^2 on launches of several waves, where rows that start on whole
sectors and rows that do not take different kernels: both give the bits that
each of the outputs has alone, and counts as the oracle's on sampled rows."""
import numpy as np
import pytest
import torch

import oracle
from qld_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [api.R2_EXACT, api.R2_REFERENCE], ids=["exact", "reference"])
@pytest.mark.parametrize("K", [2, 39, 40, 100])
@pytest.mark.parametrize("m,n", [(5003, None), (4101, 4805)])
def test_odd_and_even_rows(gpu_ctx, m, n, K, mode):
    dev, S, single = torch.device("cuda", 0), 64 * K, n is None
    n = m if single else n
    g = torch.Generator(device=dev).manual_seed(m + K)
    T = torch.randint(-2**63, 2**63 - 1, (m if single else m + n, K + (K & 1)), device=dev,
                      generator=g)
    if K & 1:
        T[:, -1] = 0
    T[7], T[m - 3, :K] = 0, -1
    bc = synth.popcount_rows(T).to(torch.int32)
    gpu_ctx.set_option(api.OPT_R2_MODE, mode)
    st = torch.cuda.current_stream()

    def run(ld, counts):
        r2 = torch.full((n, ld), -1.0, device=dev)
        cnt = torch.full((n, ld), -1, dtype=torch.int32, device=dev) if counts else None
        gpu_ctx.ld_device(T[:m], bc[:m], m, T.shape[1], None if single else T[m:],
                          None if single else bc[m:], n, T.shape[1], K, S, single, r2, ld,
                          counts=cnt, ldc=ld if counts else 0, stream=st)
        gpu_ctx.sync(st)
        return r2[:, :m].contiguous(), None if cnt is None else cnt[:, :m].contiguous()

    plain, _ = run(m, False)
    even, odd = run((m + 7) // 8 * 8, True), run((m + 7) // 8 * 8 + 1, True)
    assert torch.equal(even[0].view(torch.int32), plain.view(torch.int32))
    assert torch.equal(odd[0].view(torch.int32), plain.view(torch.int32))
    assert torch.equal(even[1], odd[1])
    host = T[:, :K].cpu().numpy().view(np.uint64)
    A, B = host[:m], host[:m] if single else host[m:]
    for b in (0, 7, n // 2, n - 1):
        want = oracle.counts(A, B[b:b + 1])[0].astype(np.int32)
        first = b if single else 0
        assert np.array_equal(odd[1][b].cpu().numpy()[first:], want[first:])
