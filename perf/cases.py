"""The work a user of qld_b200 has it do, as cases that can be timed and checked.

Every case is one call of a public entry point of ``qld_b200.api`` on the data
that call meets in use.  Tables are packed SNP rows (``qld_b200.synth``): the
haplotype-copying model for regions and bands, iid rows for task mixes.  Every
row is polymorphic, as the VCF -> MDF conversion leaves it.

Kinds:
  region   one region's lower triangle, tables and r^2 on the device
  pair     two regions' rectangle, tables and r^2 (and counts) on the device
  band     one region's windowed LD, on the device
  batch    many tasks of uneven sizes in one batched call, on the device
  hits     one region's reportable pairs (r2limit), host table to host lists
  host     two regions' rectangle, host tables to a host r^2 array
  states   joint-state codes of one region's pairs, on the device
  vcf      VCF sample fields on the host to packed rows on the host
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from qld_b200 import api, host_api, synth

R2_MODE = {"exact": api.R2_EXACT, "reference": api.R2_REFERENCE}
R2_LIMIT = 0.2          # the reportable r^2 of qLD-compute's own default runs

_contexts = {}          # one context per r^2 mode, as a program keeps it


def listed():
    return [
        # A candidate gene in a small cohort: the smallest call, latency only.
        dict(name="region_gene", kind="region", m=200, samples=1000, r2="exact", counts=False),
        # Two genes against each other in a 1000-Genomes-sized cohort, in the
        # reference's own r^2 arithmetic.
        dict(name="pair_genes", kind="pair", m=731, n=530, samples=5008, r2="reference",
             counts=False),
        # One locus, all pairs: an ordinary interactive call.
        dict(name="region_locus", kind="region", m=2048, samples=4096, r2="exact", counts=False),
        # A whole viral-genome table, all pairs: the largest ordinary call.
        dict(name="region_full", kind="region", m=29817, samples=16622, r2="exact", counts=False),
        # Two chromosome arms against each other, reference arithmetic, with
        # the joint counts kept for another statistic.
        dict(name="pair_arms", kind="pair", m=9001, n=7003, samples=16622, r2="reference",
             counts=True),
        # A chromosome in a sliding window of 1,000 SNPs (pruning, clumping).
        dict(name="band_narrow", kind="band", m=50000, band=1000, samples=10001, r2="exact"),
        # A stretch of a biobank chromosome in a wide window: long rows.
        dict(name="band_wide", kind="band", m=24000, band=5000, samples=100000, r2="exact"),
        # A task list over genes of many cohorts, one batched call.
        dict(name="batch_mix", kind="batch", tasks=300, side=2048, sizes=17, r2="exact"),
        # The report's path: one region, only its pairs above the limit leave.
        dict(name="hits_report", kind="hits", m=6001, samples=5008, r2="reference"),
        # The drop-in call on host buffers, every r^2 brought back.
        dict(name="host_pair", kind="host", m=5000, n=8001, samples=5008, r2="exact"),
        # qLD's COUNTSTATES mode on a region.
        dict(name="states_region", kind="states", m=4001, samples=16622),
        # One part of a phased 1000-Genomes chromosome, converted to rows.
        dict(name="vcf_part", kind="vcf", sites=2000, samples=2504, depth=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["region", "region", "pair", "pair", "band", "batch", "hits", "host",
                       "states", "vcf"])
    r2 = rng.choice(["exact", "reference"])
    if kind == "region":
        return dict(kind=kind, m=_log_int(rng, 64, 12000), samples=_log_int(rng, 300, 50000),
                    r2=r2, counts=rng.random() < 0.25)
    if kind == "pair":
        return dict(kind=kind, m=_log_int(rng, 64, 10000), n=_log_int(rng, 64, 10000),
                    samples=_log_int(rng, 300, 50000), r2=r2, counts=rng.random() < 0.25)
    if kind == "band":
        band = _log_int(rng, 100, 5000)
        samples = _log_int(rng, 1000, 100000)
        top = min(60000, int(1.2e13 / (band * samples)))
        return dict(kind=kind, m=_log_int(rng, 2000, max(2001, top)), band=band, samples=samples,
                    r2=r2)
    if kind == "batch":
        return dict(kind=kind, tasks=_log_int(rng, 8, 400), side=_log_int(rng, 256, 2048),
                    sizes=rng.randrange(1 << 20), r2=r2)
    if kind == "hits":
        return dict(kind=kind, m=_log_int(rng, 100, 6000), samples=_log_int(rng, 300, 20000),
                    r2=r2)
    if kind == "host":
        return dict(kind=kind, m=_log_int(rng, 100, 6000), n=_log_int(rng, 100, 6000),
                    samples=_log_int(rng, 300, 20000), r2=r2)
    if kind == "states":
        return dict(kind=kind, m=_log_int(rng, 64, 4001), samples=_log_int(rng, 300, 16622))
    return dict(kind=kind, sites=_log_int(rng, 20, 2000), samples=_log_int(rng, 200, 2504),
                depth=rng.random() < 0.5)


# ---------------------------------------------------------------- inputs --

def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _context(case):
    mode = case.get("r2", "exact")
    if mode not in _contexts:
        ctx = api.Context(torch.cuda.current_device())
        ctx.set_option(api.OPT_R2_MODE, R2_MODE[mode])
        _contexts[mode] = ctx
    return _contexts[mode]


def _polymorphic(table, samples):
    """Rows without or with only the second allele get one sample changed."""
    bc = synth.popcount_rows(table)
    first = torch.zeros_like(table[:, 0])
    first[:] = -(1 << 63)                       # sample 0 is the first word's top bit
    table[:, 0] = torch.where(bc == 0, table[:, 0] | first, table[:, 0])
    table[:, 0] = torch.where(bc == samples, table[:, 0] & ~first, table[:, 0])
    bc = torch.where(bc == 0, bc + 1, torch.where(bc == samples, bc - 1, bc))
    return table, bc.to(torch.int32)


def _copying(m, samples, seed):
    """(m, K) rows of the copying model and their bit counts."""
    dev = _device()
    f = synth.beta_freqs(m, 0.1, 1.0, seed, dev, clip_min=1.0 / samples)
    return _polymorphic(synth.copying_table(m, samples, 20, 50, 500, 0.01, f, seed, dev), samples)


def _iid(m, samples, seed):
    dev = _device()
    f = synth.beta_freqs(m, 0.5, 0.5, seed, dev).clamp(0.01, 0.99)   # a usual frequency filter
    chunk = max(64, int(2e8) // samples)
    return _polymorphic(synth.iid_table(m, samples, f, seed, dev, chunk=chunk), samples)


def _padded(table):
    """Device rows start 16-byte aligned: an even number of words apart."""
    m, K = table.shape
    if K % 2 == 0:
        return table.contiguous(), K
    out = torch.zeros(m, K + 1, dtype=torch.int64, device=table.device)
    out[:, :K] = table
    return out, K + 1


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


def _to_host(table):
    out = _pinned(table.shape, table.dtype)
    out.copy_(table)
    return out


def _tasks(case):
    """The sizes of a batched call's tasks: even ones single regions, odd ones
    two regions, as (m, n, samples, symmetric)."""
    rng = random.Random(case["sizes"])
    tasks = []
    for j in range(case["tasks"]):
        m, n = _log_int(rng, 64, case["side"]), _log_int(rng, 64, case["side"])
        samples = _log_int(rng, 1000, 50000)
        tasks.append((m, m if j % 2 == 0 else n, samples, j % 2 == 0))
    return tasks


def _batch_tables(case, seed):
    for j, (m, n, samples, symmetric) in enumerate(_tasks(case)):
        table, bc = _iid(m if symmetric else m + n, samples, seed * 1009 + j)
        yield m, n, samples, symmetric, table, bc


def _vcf_text(case, seed):
    """One part's lines from their first sample field: text, sites."""
    rng = np.random.default_rng(seed)
    sites, samples = case["sites"], case["samples"]
    freq = np.clip(rng.beta(0.3, 1.0, sites), 0.005, 0.995)
    alt = rng.random((sites, samples, 2), np.float32) < freq[:, None, None].astype(np.float32)
    width = 7 if case["depth"] else 4           # "0|1\t" or "0|1:23\t"
    text = np.empty((sites, samples, width), np.uint8)
    text[:, :, 0] = alt[:, :, 0] + ord("0")
    text[:, :, 1] = ord("|")
    text[:, :, 2] = alt[:, :, 1] + ord("0")
    if case["depth"]:
        d = rng.integers(10, 60, (sites, samples), np.uint8)
        text[:, :, 3] = ord(":")
        text[:, :, 4] = d // 10 + ord("0")
        text[:, :, 5] = d % 10 + ord("0")
    text[:, :, -1] = ord("\t")
    text[:, -1, -1] = ord("\n")
    rows = np.zeros(sites, host_api.VCF_SITE)
    rows["off"] = np.arange(sites, dtype=np.int64) * (samples * width)
    rows["len"] = samples * width - 1
    rows["n_states"] = 2
    rows["states"] = rng.choice(np.array([b"AC", b"AG", b"CT", b"GT"]), sites)
    return text.tobytes(), rows


def prepare(case, seed):
    kind, dev = case["kind"], _device()
    if kind == "vcf":
        text, sites = _vcf_text(case, seed)
        return dict(kind=kind, ctx=_context(case), text=text, sites=sites,
                    valid=np.ones(case["samples"], np.uint8), K=synth.words_for(2 * case["samples"]))
    ctx, st = _context(case), dict(kind=kind)
    if kind == "batch":
        jobs, spans, end = [], [], 0
        for m, n, samples, symmetric, table, bc in _batch_tables(case, seed):
            rows, ld = _padded(table)
            jobs.append(dict(A=rows[:m], bcA=bc[:m], m=m, lda=ld, K=table.shape[1], S=samples,
                             symmetric=symmetric, ldr=m))
            if not symmetric:
                jobs[-1].update(B=rows[m:], bcB=bc[m:], n=n, ldb=ld)
            spans.append((end, n * m))
            end += n * m
        r2 = torch.zeros(end, dtype=torch.float32, device=dev)
        for job, (at, size) in zip(jobs, spans):
            job["r2"] = r2[at:at + size]
        return dict(st, ctx=ctx, jobs=jobs, r2=r2)
    m, n, S = case["m"], case.get("n", 0), case["samples"]
    table, bc = _copying(m + n, S, seed)
    K = table.shape[1]
    st.update(ctx=ctx, m=m, n=n, S=S, K=K)
    if kind in ("hits", "host"):
        T, c = _to_host(table), bc.cpu().numpy().view(np.uint32)
        st.update(T=T, A=T[:m].numpy().view(np.uint64), bcA=c[:m])
        if kind == "hits":                      # the caller's list of values, room for all pairs
            st["val"] = np.zeros(m * (m - 1) // 2, np.float32)
        if kind == "host":
            out = _pinned((n, m), torch.float32)
            st.update(B=T[m:].numpy().view(np.uint64), bcB=c[m:], out=out, r2=out.numpy())
        return st
    rows, ld = _padded(table)
    st.update(A=rows[:m], bcA=bc[:m], B=rows[m:], bcB=bc[m:], ld=ld)
    if kind == "states":
        st["out"] = torch.zeros(m, m, dtype=torch.uint8, device=dev)
        return st
    shape = (m, case["band"]) if kind == "band" else (n or m, m)
    st["r2"] = torch.zeros(shape, dtype=torch.float32, device=dev)
    st["counts"] = torch.zeros(shape, dtype=torch.int32, device=dev) if case.get("counts") else None
    st["band"] = case.get("band")
    return st


# ------------------------------------------------------------------- run --

def run(st):
    kind, ctx = st["kind"], st["ctx"]
    if kind == "vcf":
        words, bc, length, keep = ctx.vcf_pack(st["text"], st["sites"], st["valid"], 2, st["K"])
        return dict(words=words.view(np.int64), bc=bc.view(np.int32), length=length, keep=keep)
    if kind == "hits":
        mask, row_off, val = ctx.ld_hits(st["A"], st["bcA"], S=st["S"], r2limit=R2_LIMIT)
        st["val"][:val.size] = val
        return dict(mask=mask.view(np.int32), row_off=row_off, val=st["val"])
    if kind == "host":
        return ctx.ld(st["A"], st["bcA"], st["B"], st["bcB"], S=st["S"], r2_out=st["r2"])
    stream = torch.cuda.current_stream()
    if kind == "batch":
        ctx.ld_batch(st["jobs"], stream=stream)
        return st["r2"]
    m, n, ld, K, S = st["m"], st["n"], st["ld"], st["K"], st["S"]
    if kind == "states":
        ctx.count_states_device(st["A"], m, ld, None, m, ld, K, True, st["out"], m, stream=stream)
        return st["out"]
    if kind == "band":
        ctx.ld_band_device(st["A"], st["bcA"], m, ld, K, S, st["band"], st["r2"], st["band"],
                           stream=stream)
        return st["r2"]
    counts, ldc = st["counts"], m if st["counts"] is not None else 0
    if kind == "region":
        ctx.ld_device(st["A"], st["bcA"], m, ld, None, None, m, ld, K, S, True, st["r2"], m,
                      counts=counts, ldc=ldc, stream=stream)
    else:
        ctx.ld_device(st["A"], st["bcA"], m, ld, st["B"], st["bcB"], n, ld, K, S, False, st["r2"],
                      m, counts=counts, ldc=ldc, stream=stream)
    return st["r2"] if counts is None else dict(r2=st["r2"], counts=counts)


# ------------------------------------------------------------------ work --

def _pairs(case):
    kind, m = case["kind"], case.get("m", 0)
    if kind == "band":
        w = min(case["band"], m - 1)
        return m * w - w * (w + 1) // 2
    if kind in ("pair", "host"):
        return m * case["n"]
    return m * (m + 1) // 2


def work(case):
    kind = case["kind"]
    if kind == "vcf":
        fields = case["sites"] * case["samples"]
        out = case["sites"] * (8 * synth.words_for(2 * case["samples"]) + 9)
        return dict(bytes=fields * (7 if case["depth"] else 4) + out, flops=0)
    if kind == "batch":
        total = dict(bytes=0, flops=0)
        for m, n, samples, symmetric in _tasks(case):
            K, pairs = synth.words_for(samples), m * (m + 1) // 2 if symmetric else m * n
            rows = m if symmetric else m + n
            total["bytes"] += rows * (8 * K + 4) + 4 * pairs
            total["flops"] += 128 * K * pairs
        return total
    K, pairs, rows = synth.words_for(case["samples"]), _pairs(case), case["m"] + case.get("n", 0)
    if kind == "states":                        # one byte a pair; no arithmetic it must do
        return dict(bytes=rows * 8 * K + pairs, flops=0)
    out = 4 * pairs * (2 if case.get("counts") else 1)
    if kind == "hits":                          # a bit a pair, and the few values above the limit
        out = case["m"] * ((case["m"] + 31) // 32 * 4 + 8)
    return dict(bytes=rows * (8 * K + 4) + out, flops=128 * K * pairs)


# ----------------------------------------------------------------- exact --

def _bits(table, samples):
    """(rows, K) packed words -> (rows, samples) float64 zeros and ones."""
    shift = torch.arange(63, -1, -1, device=table.device)
    parts = [((rows.unsqueeze(2) >> shift) & 1).flatten(1)[:, :samples].to(torch.float64)
             for rows in table.split(1024)]
    return torch.cat(parts)


def _r2(joint, ca, cb, S):
    """r^2 of B rows (bit counts cb) against A rows (ca) from joint counts."""
    ca, cb = ca.to(torch.float64)[None, :], cb.to(torch.float64)[:, None]
    d = S * joint - ca * cb
    return d * d / (ca * (S - ca) * cb * (S - cb))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("hits", "states", "vcf"):       # lists whose lengths are the answer, codes, bits
        return None
    if kind == "batch":
        parts = []
        for m, n, samples, symmetric, table, bc in _batch_tables(case, seed):
            x = _bits(table, samples)
            a, b, ca, cb = (x, x, bc, bc) if symmetric else (x[:m], x[m:], bc[:m], bc[m:])
            r2 = _r2(b @ a.T, ca, cb, samples)
            parts.append((r2.triu() if symmetric else r2).flatten())
        return torch.cat(parts)
    m, n, S = case["m"], case.get("n", 0), case["samples"]
    table, bc = _copying(m + n, S, seed)
    if kind == "band":
        w, step = case["band"], 2000
        out = torch.zeros(m, w, dtype=torch.float64, device=table.device)
        for i0 in range(0, m - 1, step):
            i1, j1 = min(m, i0 + step), min(m, i0 + step + w)
            x = _bits(table[i0:j1], S)
            r2 = _r2(x[:i1 - i0] @ x.T, bc[i0:j1], bc[i0:i1], S)
            j = torch.arange(i1 - i0, device=x.device)[:, None] + 1 + torch.arange(w, device=x.device)
            inside = j < j1 - i0
            out[i0:i1] = torch.where(inside, r2.gather(1, j.clamp(max=j1 - i0 - 1)), 0.0)
        return out
    x = _bits(table, S)
    if kind == "region":
        r2 = torch.empty(m, m, dtype=torch.float64, device=x.device)
        for i in range(0, m, 4096):
            r2[i:i + 4096] = _r2(x[i:i + 4096] @ x.T, bc, bc[i:i + 4096], S)
        r2 = r2.triu_()
    else:
        r2 = _r2(x[m:] @ x[:m].T, bc[:m], bc[m:], S)
    return dict(r2=r2, counts=None) if case.get("counts") else r2
