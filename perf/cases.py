"""The searches this library is used for, as cases that can be timed.

A case names a call and its sizes: plain 2-way and 3-way searches (K2 and MI,
planes on the device or in pinned host memory, whole or one slab of the first
SNPs as one of several GPUs searches it), a batch of uneven cohorts, a batch of
phenotype permutations, and the genotype-matrix binarizer.  Data is synthetic:
Hardy-Weinberg genotypes with minor-allele frequencies uniform in
[maf_min, 0.5], cases and controls drawn with one planted set of the search's
order (P(case) 0.5, or 0.75 for carriers of a minor allele at all its SNPs).

``run`` makes one call through the Python binding of the C-ABI; ``exact``
scores every set in 64 bits with plain torch where that is quick.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensor-episdet_b200"))

import episdet  # noqa: E402
import sharded  # noqa: E402

GPU = "cuda"
BATCH = 16  # cohorts of a batch, labels of a permutation batch
MAX_WORK = 4.0e14  # sets x samples of the largest case, per call


def _search(name, order, score, snps, cases, controls, shards=1, rank=0, host=False, top_k=1024, maf_min=0.05):
    return {"name": name, "call": "search", "order": order, "score": score, "snps": snps, "cases": cases,
            "controls": controls, "shards": shards, "rank": rank, "host": host, "top_k": top_k, "maf_min": maf_min}


def listed():
    return [
        # A candidate panel against a small study: the smallest search, all latency.
        _search("pairs_k2_512x4096", 2, "k2", 512, 2048, 2048),
        # The same with uneven classes that fill no word, a short list, the other score.
        _search("pairs_mi_1000x5003", 2, "mi", 1000, 2001, 3002, top_k=100),
        # A study read from files, as the command line does it: planes in host memory.
        _search("pairs_k2_host_8192x50001", 2, "k2", 8192, 20000, 30001, host=True),
        # All pairs of a large panel.
        _search("pairs_mi_16384x32768", 2, "mi", 16384, 16384, 16384),
        # All triplets of a candidate panel, hundreds of SNPs: many small steps.
        _search("triplets_k2_256x4096", 3, "k2", 256, 2048, 2048),
        _search("triplets_mi_600x10007", 3, "mi", 600, 4003, 6004, top_k=100, maf_min=0.01),
        # All triplets of a mid-size panel.
        _search("triplets_k2_1536x40000", 3, "k2", 1536, 16000, 24000),
        # One GPU's share (of eight) of the 4,096 x 262,144 search: the largest study.
        _search("triplets_k2_4096x262144_r3of8", 3, "k2", 4096, 131072, 131072, shards=8, rank=3),
        # One share of sixteen of the 8,192 x 65,536 MI search: many SNPs, rare alleles.
        _search("triplets_mi_8192x65536_r5of16", 3, "mi", 8192, 32768, 32768, shards=16, rank=5, maf_min=0.01),
        # Uneven cohorts in one call, half of them 2-way and half 3-way.
        {"name": "batched_16_cohorts", "call": "batched", "score": "k2", "snps_min": 256, "snps_max": 1024,
         "samples_min": 4096, "samples_max": 131072, "maf_min": 0.05, "shape_seed": 4},
        # Significance by permutation: the observed labels and 15 shuffled ones.
        {"name": "perm_k2_16384x32768_16", "call": "perm", "score": "k2", "snps": 16384, "samples": 32768,
         "cases": 16384, "top_k": 1024, "maf_min": 0.05},
        # A genotype matrix made into bit planes before a search.
        {"name": "binarize_8192x50001", "call": "binarize", "snps": 8192, "cases": 20000, "controls": 30001,
         "maf_min": 0.05},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["pairs", "pairs", "triplets", "triplets", "triplets", "batched", "perm", "binarize"])
    score = rng.choice(["k2", "mi"])
    maf_min = rng.choice([0.01, 0.05])
    n = _log_uniform(rng, 2000, 262144 if call == "triplets" else 65536)
    cases = max(1, int(n * rng.uniform(0.3, 0.7)))
    if call == "batched":
        return {"call": "batched", "score": score, "snps_min": rng.choice([128, 256]), "snps_max": 1024,
                "samples_min": 2000, "samples_max": 100000, "maf_min": maf_min, "shape_seed": rng.randrange(1 << 20)}
    if call == "perm":
        snps = _log_uniform(rng, 512, 12000)
        return {"call": "perm", "score": score, "snps": snps, "samples": min(n, 32768), "cases": min(cases, 16000),
                "top_k": rng.choice([1, 100, 1024]), "maf_min": maf_min}
    if call == "binarize":
        return {"call": "binarize", "snps": _log_uniform(rng, 512, 8192), "cases": cases, "controls": n - cases,
                "maf_min": maf_min}
    order = 2 if call == "pairs" else 3
    snps = _log_uniform(rng, 300, 16384) if order == 2 else _log_uniform(rng, 128, 6000)
    shards = max(1, math.ceil(math.comb(snps, order) * n / (0.5 * MAX_WORK)))
    case = _search(None, order, score, snps, cases, n - cases, shards=shards, rank=rng.randrange(shards),
                   host=rng.random() < 0.25, top_k=rng.choice([1, 100, 1024, 1024, 1536]), maf_min=maf_min)
    del case["name"]
    return case


# ------------------------------------------------------------------ data
def _pack(bits):
    """Boolean [rows][n] -> int32 words [rows][ceil(n/1024)*32], first sample in the top bit."""
    rows, n = bits.shape
    padded = torch.zeros((rows, episdet.class_words(n) * 32), dtype=torch.bool, device=bits.device)
    padded[:, :n] = bits
    weights = 2 ** torch.arange(7, -1, -1, dtype=torch.int32, device=bits.device)
    octets = (padded.view(rows, -1, 8) * weights).sum(-1, dtype=torch.int32).view(rows, -1, 4)
    return (octets[..., 0] << 24) | (octets[..., 1] << 16) | (octets[..., 2] << 8) | octets[..., 3]


def _genotypes(maf, n, gen):
    """[len(maf)][n] genotypes 0/1/2 (minor-allele counts), Hardy-Weinberg."""
    u = torch.rand((len(maf), n), generator=gen, device=GPU)
    q = 1.0 - maf[:, None]
    return (u >= q * q).to(torch.uint8) + (u >= q * q + 2.0 * q * maf[:, None]).to(torch.uint8)


def _planted(maf, cases, controls, gen):
    """Genotypes of the planted SNPs in the cases and in the controls."""
    n = 4 * max(cases, controls) + 4096
    g = _genotypes(maf, n, gen)
    risk = 0.5 + 0.25 * (g > 0).all(0).float()
    is_case = torch.rand(n, generator=gen, device=GPU) < risk
    return g[:, is_case][:, :cases], g[:, ~is_case][:, :controls]


def _class_genotypes(snps, cases, controls, order, maf_min, seed):
    """Yields (first row, genotypes) blocks of the cases and of the controls."""
    gen = torch.Generator(device=GPU).manual_seed(seed)
    maf = maf_min + (0.5 - maf_min) * torch.rand(snps, generator=gen, device=GPU)
    sets = sorted(int(v) for v in torch.randperm(snps, generator=gen, device=GPU)[:order].tolist())
    maf[sets] = 0.25
    special = _planted(maf[sets], cases, controls, gen)
    step = max(1, min(snps, (1 << 26) // max(cases, controls)))
    for r0 in range(0, snps, step):
        block = maf[r0:r0 + step]
        for c, n in enumerate((cases, controls)):
            g = _genotypes(block, n, gen)
            for i, s in enumerate(sets):
                if r0 <= s < r0 + step:
                    g[s - r0] = special[c][i]
            yield c, r0, g


def _planes(snps, cases, controls, order, maf_min, seed):
    out = [torch.zeros((snps, 2, episdet.class_words(n)), dtype=torch.int32, device=GPU) for n in (cases, controls)]
    for c, r0, g in _class_genotypes(snps, cases, controls, order, maf_min, seed):
        for v in range(2):
            out[c][r0:r0 + len(g), v] = _pack(g == v)
    return out


def _cohort_shapes(case):
    rng = np.random.default_rng(case["shape_seed"])
    out = []
    for i in range(BATCH):
        m = int(round(math.exp(rng.uniform(math.log(case["snps_min"]), math.log(case["snps_max"])))))
        n = int(round(math.exp(rng.uniform(math.log(case["samples_min"]), math.log(case["samples_max"])))))
        nc = int(round(n * rng.uniform(0.3, 0.7)))
        out.append((m, nc, n - nc, 2 + i % 2))
    return out


def _labels(samples, cases, seed):
    gen = torch.Generator(device=GPU).manual_seed(seed)
    bits = torch.zeros((BATCH, samples), dtype=torch.bool, device=GPU)
    bits[0, :cases] = True
    for i in range(1, BATCH):
        bits[i, torch.randperm(samples, generator=gen, device=GPU)[:cases]] = True
    return bits


def _slab(case):
    if case["shards"] == 1:
        return 0, 0
    return sharded.work_slabs(case["snps"], case["order"], case["shards"])[case["rank"]]


def prepare(case, seed):
    call = case["call"]
    if call == "search":
        planes = _planes(case["snps"], case["cases"], case["controls"], case["order"], case["maf_min"], seed)
        if case["host"]:
            planes = [p.cpu().pin_memory() for p in planes]
        begin, end = _slab(case)
        return {"case": case, "planes": planes, "begin": begin, "end": end}
    if call == "batched":
        cohorts, options = [], []
        for i, (m, nc, nn, order) in enumerate(_cohort_shapes(case)):
            a, b = _planes(m, nc, nn, order, case["maf_min"], seed * BATCH + i)
            cohorts.append((a, b, nc, nn, m))
            options.append({"order": order, "score": case["score"]})
        return {"case": case, "cohorts": cohorts, "options": options}
    if call == "perm":
        # The observed cases are the first samples; the other labels shuffle them.
        a = torch.zeros((case["snps"], 2, episdet.class_words(case["samples"])), dtype=torch.int32, device=GPU)
        parts = {}
        for c, r0, g in _class_genotypes(case["snps"], case["cases"], case["samples"] - case["cases"], 2,
                                         case["maf_min"], seed):
            parts[c] = g
            if c == 1:
                both = torch.cat([parts[0], parts[1]], 1)
                for v in range(2):
                    a[r0:r0 + len(g), v] = _pack(both == v)
        return {"case": case, "planes": a, "labels": _pack(_labels(case["samples"], case["cases"], seed))}
    n = case["cases"] + case["controls"]
    geno = torch.empty((case["snps"], n), dtype=torch.uint8, device=GPU)
    gen = torch.Generator(device=GPU).manual_seed(seed + 1)
    order = torch.randperm(n, generator=gen, device=GPU)
    flags = torch.zeros(n, dtype=torch.uint8, device=GPU)
    flags[order[:case["cases"]]] = 1
    columns = (order[:case["cases"]], order[case["cases"]:])
    for c, r0, g in _class_genotypes(case["snps"], case["cases"], case["controls"], 2, case["maf_min"], seed):
        geno[r0:r0 + len(g), columns[c]] = g
    return {"case": case, "genotypes": geno, "flags": flags}


# ------------------------------------------------------------------ the calls
def _result(r):
    return {"score": r.score, "top_snps": r.top_snps.astype(np.int64), "top_fp32": r.top_fp32, "top_fp64": r.top_fp64}


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "search":
        return _result(episdet.search(state["planes"][0], state["planes"][1], case["cases"], case["controls"],
                                      order=case["order"], score=case["score"], top_k=case["top_k"],
                                      first_begin=state["begin"], first_end=state["end"]))
    if call == "batched":
        return [_result(r) for r in episdet.search_batched(state["cohorts"], state["options"])]
    if call == "perm":
        return [_result(r) for r in episdet.search_perm(state["planes"], case["samples"], state["labels"],
                                                        score=case["score"], top_k=case["top_k"])]
    cases, controls, nc, nn = episdet.binarize(state["genotypes"], state["flags"])
    return {"cases": cases, "controls": controls, "num_cases": nc, "num_controls": nn}


# ------------------------------------------------------------------ work
def _sets(order, snps, begin=0, end=0):
    return sum(math.comb(snps - 1 - x, order - 1) for x in range(begin, min(end or snps, snps)))


def _plane_bytes(snps, *classes):
    return sum(8 * snps * episdet.class_words(n) for n in classes)


def _search_work(order, snps, cases, controls, begin=0, end=0):
    # A pair needs 4 counts over all samples; a triplet needs 4 over the samples
    # of the first SNP's two rarer genotypes (about half of them), the rest
    # following from pair counts.
    n = cases + controls
    per_set = 2.0 * 4 * n * (1.0 if order == 2 else 0.5)
    return {"bytes": _plane_bytes(snps, cases, controls), "flops": _sets(order, snps, begin, end) * per_set}


def work(case):
    call = case["call"]
    if call == "search":
        begin, end = _slab(case)
        return _search_work(case["order"], case["snps"], case["cases"], case["controls"], begin, end)
    if call == "batched":
        parts = [_search_work(o, m, nc, nn) for m, nc, nn, o in _cohort_shapes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if call == "perm":
        # All pairs over all samples once, then over the cases of each label.
        pairs = _sets(2, case["snps"])
        return {"bytes": _plane_bytes(case["snps"], case["samples"]),
                "flops": 2.0 * 4 * pairs * (case["samples"] + BATCH * case["cases"])}
    n = case["cases"] + case["controls"]
    return {"bytes": case["snps"] * n + _plane_bytes(case["snps"], case["cases"], case["controls"]), "flops": 0}


# ------------------------------------------------------------------ 64-bit check
def _onehot(planes, n):
    """int32 planes [M][2][W] -> float32 indicator rows [3 M][n] of genotypes 0, 1, 2."""
    m = planes.shape[0]
    out = torch.empty((m, 3, n), dtype=torch.float32, device=GPU)
    shift = torch.arange(31, -1, -1, dtype=torch.int32, device=GPU)
    step = max(1, (1 << 26) // max(1, n))
    for r0 in range(0, m, step):
        bits = ((planes[r0:r0 + step].to(GPU)[..., None] >> shift) & 1).flatten(2)[..., :n].float()
        out[r0:r0 + step, :2] = bits
        out[r0:r0 + step, 2] = 1.0 - bits.sum(1)
    return out.view(3 * m, n)


class _Scores:
    """64-bit scores of tables whose cells are the last axis, and the best k of all that were offered."""

    def __init__(self, score, cases, controls, k):
        n = cases + controls
        v = torch.arange(n + 2, dtype=torch.float64, device=GPU)
        self.mi, self.k, self.best = score == "mi", k, None
        self.cases, self.controls, self.n = cases, controls, n
        self.table = (v / n) * torch.log2(torch.clamp(v, min=1.0) / n) if self.mi else torch.lgamma(v + 1.0)

    def offer(self, cs, cn, mask):
        """cs, cn: long [..., cells]; only sets under mask count."""
        t = self.table
        if self.mi:
            hy = -sum(c / self.n * math.log2(c / self.n) for c in (self.cases, self.controls))
            s = hy + (t[cs] + t[cn] - t[cs + cn]).sum(-1)
        else:
            s = (t[cs] + t[cn] - t[cs + cn + 1]).sum(-1).abs()
        s = s[mask] if not self.mi else -s[mask]
        s = s if self.best is None else torch.cat([self.best, s])
        self.best = torch.topk(s, min(self.k, len(s)), largest=False).values.sort().values if len(s) else None

    def result(self):
        top = (-self.best if self.mi else self.best).cpu().numpy()
        # The list is in the order of the 32-bit scores, the same up to their rounding.
        return {"score": float(top[0]), "top_snps": None, "top_fp32": top, "top_fp64": top}


def _cells(a, b, m):
    """Counts of a block's indicator rows [3 k][n] against all [3 m][n]: long [k][m][9]."""
    c = a @ b.T
    return c.view(-1, 3, m, 3).permute(0, 2, 1, 3).reshape(-1, m, 9).long()


def _exact_pairs(rows, m, scores, total=None):
    step = max(1, (1 << 22) // m)
    z = torch.arange(m, device=GPU)
    for a0 in range(0, m, step):
        k = min(step, m - a0)
        cs = _cells(rows[0][3 * a0:3 * (a0 + k)], rows[0], m)
        cn = _cells(rows[1][3 * a0:3 * (a0 + k)], rows[1], m) if total is None else total[a0:a0 + k].long() - cs
        scores.offer(cs, cn, z[None, :] > torch.arange(a0, a0 + k, device=GPU)[:, None])


def _exact_triplets(rows, m, scores, begin, end):
    z = torch.arange(m, device=GPU)
    for x in range(begin, min(end or m, m - 2)):
        tabs = [torch.cat([_cells(r[3 * x + 3:] * r[3 * x + g], r[3 * x + 3:], m - x - 1) for g in range(3)], -1)
                for r in rows]
        zz = z[x + 1:]
        scores.offer(tabs[0], tabs[1], zz[None, :] > zz[:, None])


def _exact_search(order, score, planes, cases, controls, top_k, begin=0, end=0):
    m = planes[0].shape[0]
    flops = 18.0 * m * m * (cases + controls) * (1 if order == 2 else (min(end or m, m) - begin))
    if flops > 1.5e15 or (order == 3 and _sets(3, m, begin, end) > 3e8):
        return None
    rows = [_onehot(p, n) for p, n in zip(planes, (cases, controls))]
    scores = _Scores(score, cases, controls, top_k)
    if order == 2:
        _exact_pairs(rows, m, scores)
    else:
        _exact_triplets(rows, m, scores, begin, end)
    return scores.result()


def exact(case, seed):
    """Indicator products are whole numbers below 2^24: exact in 32-bit sums, TF32 inputs too."""
    tf32 = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        return _exact(case, prepare(case, seed))
    finally:
        torch.backends.cuda.matmul.allow_tf32 = tf32


def _exact(case, state):
    call = case["call"]
    if call == "search":
        return _exact_search(case["order"], case["score"], state["planes"], case["cases"], case["controls"],
                             case["top_k"], state["begin"], state["end"])
    if call == "batched":
        return [_exact_search(opt["order"], case["score"], co[:2], co[2], co[3], 1024)
                for co, opt in zip(state["cohorts"], state["options"])]
    if call == "perm":
        m, n, k = case["snps"], case["samples"], case["cases"]
        rows = _onehot(state["planes"], n)
        total = torch.empty((m, m, 9), dtype=torch.int32, device=GPU)
        step = max(1, (1 << 22) // m)
        for a0 in range(0, m, step):
            total[a0:a0 + step] = _cells(rows[3 * a0:3 * (a0 + step)], rows, m)
        out = []
        for label in _label_bits(state["labels"], n):
            scores = _Scores(case["score"], k, n - k, case["top_k"])
            _exact_pairs([rows[:, label]], m, scores, total)
            out.append(scores.result())
        return out
    return None


def _label_bits(labels, n):
    shift = torch.arange(31, -1, -1, dtype=torch.int32, device=GPU)
    return ((labels[..., None] >> shift) & 1).flatten(1)[:, :n].bool()
