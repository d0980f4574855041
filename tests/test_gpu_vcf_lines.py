"""VCF packing of lines shorter and longer than the staging buffer, phased,
unphased and mixed, with other subfields, runs of separators and line ends,
against the oracle."""
import numpy as np
import pytest

import oracle
from qld_b200 import host_api

pytestmark = pytest.mark.gpu


def _lines(sites, samples, seed, kinds):
    """Text and records of `sites` lines of `samples` fields of mixed kinds."""
    rng = np.random.default_rng(seed)
    rows = np.zeros(sites, host_api.VCF_SITE)
    text = b""
    for i in range(sites):
        kind = kinds[i % len(kinds)]
        g = rng.integers(0, 2, (samples, 2))
        bar = {"phased": "|", "unphased": "/"}.get(kind, "|")
        fields = [f"{a}{bar}{b}" for a, b in g]
        if kind == "depth":
            fields = [f"{f}:{rng.integers(1000)}" for f in fields]
        elif kind == "mixed":
            fields = [f.replace("|", "/") if rng.random() < 0.1 else f for f in fields]
        elif kind == "missing":
            fields = [".|." if rng.random() < 0.01 else f for f in fields]
        elif kind == "second":
            fields = [f"{rng.integers(9)}:{f}" for f in fields]
        sep = [" \t" if rng.random() < 0.02 else "\t" for _ in fields]
        line = "".join(s + f for s, f in zip(sep[1:], fields[1:]))
        line = (" " if i % 3 == 1 else "") + fields[0] + line + ("\t" if i % 4 == 2 else "")
        text += b"x" * int(rng.integers(1, 18))          # any alignment of the first field
        rows[i] = (len(text), len(line), 1 if kind == "second" else 0, 2, b"AG")
        text += line.encode() + b"\n"
    return text, rows


@pytest.mark.parametrize("sites,samples", [(60, 3), (40, 65), (30, 700), (6, 12100)])
@pytest.mark.parametrize("kinds", [("phased", "depth"), ("unphased",),
                                   ("phased", "mixed", "missing", "second", "unphased")])
def test_lines_equal_oracle(gpu_ctx, sites, samples, kinds):
    text, rows = _lines(sites, samples, sites + samples, kinds)
    valid = np.ones(samples, np.uint8)
    valid[::7] = 0
    K = (2 * int(valid.sum()) + 63) // 64
    oracle.vcf_seed(1)
    want = oracle.vcf_pack(text, rows, valid, 2, K)
    got = gpu_ctx.vcf_pack(text, rows, valid, 2, K, seed=1)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
