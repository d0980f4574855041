"""COUNTSTATES evaluated from the end of the rows (ld_states.cu): rows that
settle at once, late, or only at the start, against the oracle's fold."""
import numpy as np
import pytest

import oracle
from qld_b200 import synth

pytestmark = pytest.mark.gpu

FULL = np.uint64(0xFFFFFFFFFFFFFFFF)


def _rows(m, K, seed):
    """Rows of every kind the shortcuts look at, in random order."""
    rng = np.random.default_rng(seed)
    T = np.zeros((m, K), np.uint64)
    for r in range(m):
        kind = r % 8
        if kind == 1:                                  # one bit somewhere
            T[r, rng.integers(K)] = np.uint64(1) << np.uint64(rng.integers(64))
        elif kind == 2:                                # all ones, or all but one word
            T[r] = FULL
            if rng.random() < 0.5:
                T[r, rng.integers(K)] = 0
        elif kind == 3:                                # a run of ones at one end
            k = int(rng.integers(K + 1))
            T[r, :k] = FULL
            if rng.random() < 0.5:
                T[r] = T[r, ::-1]
        elif kind == 4:                                # full words and empty words
            T[r] = np.where(rng.random(K) < 0.5, FULL, np.uint64(0))
        elif kind == 5:                                # halves that add up to 64 with others
            T[r] = np.uint64(0x00000000FFFFFFFF) << np.uint64(32 * rng.integers(2))
        elif kind == 6:                                # a few bits
            T[r, rng.integers(0, K, 3)] = rng.integers(1, 1 << 63, 3, dtype=np.uint64)
        elif kind == 7:
            T[r] = rng.integers(0, 1 << 64, K, dtype=np.uint64)
    return T[rng.permutation(m)]


@pytest.mark.parametrize("K", [1, 7, 8, 9, 33, 72, 129, 300])
def test_every_kind_of_row(gpu_ctx, K):
    T = _rows(330, K, K)
    A, B = T[:190], T[190:]
    assert np.array_equal(gpu_ctx.count_states(A, B), oracle.count_states(A, B))


def test_rare_alleles_long_rows(gpu_ctx):
    f = synth.beta_freqs(300, 0.05, 2.0, 5, clip_min=1.0 / 30000)
    T = synth.iid_table(300, 30000, f, 5).numpy().view(np.uint64)
    got, want = gpu_ctx.count_states(T), oracle.count_states(T)
    keep = np.arange(300)[None, :] >= np.arange(300)[:, None]
    assert np.array_equal(got[keep], want[keep])
