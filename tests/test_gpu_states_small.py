"""COUNTSTATES of short rows and of tables at the edges of a tile, where the
whole fold is one walk or little more, against the oracle; entries that a task
does not owe stay as they were."""
import numpy as np
import pytest
import torch

import oracle
from test_gpu_states_suffix import _rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 6, 7, 9])
@pytest.mark.parametrize("m,n", [(1, None), (31, None), (33, None), (127, None), (128, None),
                                 (130, None), (301, None), (1, 300), (129, 15), (96, 129),
                                 (400, 17)])
def test_short_rows(gpu_ctx, m, n, K):
    single = n is None
    n = m if single else n
    T = _rows(m if single else m + n, K, 100 * K + m)
    A, B = T[:m], T[:m] if single else T[m:]
    lda = K + (K & 1)
    D = torch.zeros(T.shape[0], lda, dtype=torch.int64, device="cuda")
    D[:, :K] = torch.from_numpy(T.view(np.int64)).cuda()
    out = torch.full((n, m + 5), 99, dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream()
    gpu_ctx.count_states_device(D[:m], m, lda, None if single else D[m:].contiguous(), n, lda, K,
                                single, out, m + 5, stream=st)
    gpu_ctx.sync(stream=st)
    got = out.cpu().numpy()
    keep = np.arange(m)[None, :] >= np.arange(n)[:, None] if single else np.ones((n, m), bool)
    assert np.array_equal(got[:, :m][keep], oracle.count_states(A, B)[keep])
    assert np.all(got[:, m:] == 99) and np.all(got[:, :m][~keep] == 99)
