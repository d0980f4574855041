"""COUNTSTATES of a single region streamed in blocks of B rows (each block's
tiles start below its own part of the diagonal), against the oracle."""
import numpy as np
import pytest

import oracle
from qld_b200 import api
from test_gpu_states_suffix import _rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,K", [(257, 3), (511, 5), (700, 6), (1030, 13), (1290, 40)])
def test_single_region_in_blocks(gpu_ctx, m, K):
    T = _rows(m, K, m)
    want = oracle.count_states(T)
    keep = np.arange(m)[None, :] >= np.arange(m)[:, None]
    for rows in (256, 512):
        gpu_ctx.set_option(api.OPT_BAND_ROWS, rows)
        try:
            got = gpu_ctx.count_states(T)
        finally:
            gpu_ctx.set_option(api.OPT_BAND_ROWS, 4096)
        assert np.array_equal(got[keep], want[keep])
