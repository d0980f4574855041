"""VCF packing of lines about as long as the staging buffer holds (47 KB), and of
short and longer ones in one call, phased and not, against the oracle."""
import numpy as np
import pytest

import oracle
from qld_b200 import host_api

pytestmark = pytest.mark.gpu

LIMIT = 47 * 1024


def _text(lengths, samples, seed):
    """Lines of `samples` fields padded to `lengths` bytes with a second subfield,
    each at another alignment; every third line unphased in places."""
    rng = np.random.default_rng(seed)
    rows = np.zeros(len(lengths), host_api.VCF_SITE)
    text = b""
    for i, want in enumerate(lengths):
        bars = np.where(rng.random(samples) < (0.2 if i % 3 == 2 else 0.0), "/", "|")
        fields = [f"{a}{bar}{b}" for bar, (a, b) in zip(bars, rng.integers(0, 2, (samples, 2)))]
        pad = want - (4 * samples - 1)
        if pad > 0:                      # over all fields: the oracle's words are 64 KB
            share = np.full(samples, pad // samples)
            share[:pad % samples] += 1
            fields = [f + (":" + "7" * (k - 1) if k else "") for f, k in zip(fields, share)]
        line = "\t".join(fields).encode()
        assert len(line) == max(want, 4 * samples - 1)
        text += b"#" * (i % 16 + 1)
        rows[i] = (len(text), len(line), 0, 2, b"CT")
        text += line + b"\n"
    return text, rows


@pytest.mark.parametrize("lengths", [
    [0, 0, 0, LIMIT + 5000, 0, 0],                            # one long line among short ones
    [LIMIT + 100, 0, LIMIT + 101, 2000, 300000, 0, 0, 7],     # long ones first and between
    [LIMIT - 48, LIMIT - 32] * 3, [LIMIT - 31] * 3, [LIMIT - 30] * 3,          # at the limit
    [LIMIT - 16, LIMIT - 15, LIMIT - 1, LIMIT, LIMIT + 1, LIMIT + 16] * 3,
    [LIMIT + 1] * 4])                                         # none staged
def test_long_and_short_lines(gpu_ctx, lengths):
    samples = 150
    text, rows = _text(lengths, samples, len(lengths) + lengths[-1])
    valid = np.ones(samples, np.uint8)
    valid[::9] = 0
    K = (2 * int(valid.sum()) + 63) // 64
    oracle.vcf_seed(1)
    want = oracle.vcf_pack(text, rows, valid, 2, K)
    got = gpu_ctx.vcf_pack(text, rows, valid, 2, K, seed=1)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
