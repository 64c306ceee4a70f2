"""The searches a user of this library runs, as cases to be timed: one pass of a case is one call
of a public entry point (``GpuSearch.run`` or ``GpuSearch.run_batch``) with the results taken out.

Sizes are the named workloads of ``fiuncho_gb300.synth`` and of ``bench.py``, and odd ones between
them.  Genotypes are drawn under Hardy-Weinberg equilibrium from a per-SNP minor-allele frequency,
with one planted interaction, as in ``fiuncho_gb300.synth`` (made on the GPU here, so that large
data sets are quick).
"""
import itertools
import math

import numpy as np
import torch

from fiuncho_gb300 import Dataset, Distribution, GpuSearch
from fiuncho_gb300.ingest import upload_genotypes


def _scan(name, order, snps, cases, ctrls, outputs, source="resident", maf="uniform", step=1, offset=0, missing=0.0):
    return {"name": name, "order": order, "snps": snps, "cases": cases, "ctrls": ctrls, "outputs": outputs,
            "source": source, "maf": maf, "step": step, "offset": offset, "missing": missing}


def listed():
    return [
        # a pathway's worth of SNPs, read from files and searched once: the call's own latency counts
        _scan("o3_187x997_host", 3, 187, 511, 486, 10, source="host"),
        # the plain pair search of a candidate-gene panel, host data set in, results out
        _scan("o2_1000x4000_host", 2, 1000, 2000, 2000, 10, source="host"),
        # pairs of a mid-size array kept on the device
        _scan("o2_12001x3999", 2, 12001, 1900, 2099, 100),
        # the large pair scan: rare and common variants, 8e8 pairs
        _scan("o2_40000x16000", 2, 40000, 8000, 8000, 1000, maf="beta"),
        # the headline triple search
        _scan("o3_2000x8000", 3, 2000, 4000, 4000, 100),
        # triples of a large cohort (the class sizes of the reference's own test data)
        _scan("o3_500x18800", 3, 500, 9000, 9800, 100),
        # one rank's strided share of a triple search (MPIEngine hands rank r Distribution(n, 2, size, r))
        _scan("o3_1201x6501_rank1of4", 3, 1201, 2999, 3502, 100, step=4, offset=1),
        # quadruples, the largest search a user waits for
        _scan("o4_300x8000", 4, 300, 4000, 4000, 100),
        # quadruples of a small cohort: many combinations, few samples each
        _scan("o4_300x1570", 4, 300, 558, 1012, 50),
        # quadruples of a large cohort
        _scan("o4_100x18800", 4, 100, 9000, 9800, 50),
        # data with ungenotyped calls: the full-table path
        _scan("o3_400x8000_missing", 3, 400, 4000, 4000, 100, missing=0.01),
        # many uneven scans in one call
        {"name": "batch_12_uneven", "scans": 12, "base": 77, "max_snps": 1200, "order4_cap": 150,
         "min_samples": 1000, "max_samples": 16000, "outputs": 50},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _combos(c):
    """Combinations of a scan (a strided share owns one prefix in `step`)."""
    return math.comb(c["snps"], c["order"]) / c["step"]


def _flops(c):
    """2^order core cells a combination, a multiply-add a sample each (the others follow from the marginals)."""
    return 2.0 * 2 ** c["order"] * _combos(c) * (c["cases"] + c["ctrls"])


# no drawn scan above these (the largest listed ones): combinations x samples, and combinations for
# the orders whose cost is the tables' evaluation
_MOST_WORK = {2: 1.28e13, 3: 1.06e13, 4: 2.6e12}
_MOST_COMBOS = {2: 8.0e8, 3: 1.33e9, 4: 3.3e8}
_MISSING_WORK = 8.5e10


def draw(rng):
    if rng.random() < 0.1:
        return {"scans": rng.randint(4, 12), "base": rng.randint(0, 10 ** 6), "max_snps": _log(rng, 250, 1200),
                "order4_cap": rng.randint(60, 150), "min_samples": 1000, "max_samples": _log(rng, 2000, 16000),
                "outputs": rng.randint(5, 50)}
    while True:
        order = rng.choice([2, 2, 3, 3, 3, 4, 4])
        lo, hi = {2: (300, 40000), 3: (100, 2000), 4: (50, 300)}[order]
        snps, samples = _log(rng, lo, hi), _log(rng, 900, 20000)
        cases = max(1, int(round(samples * rng.uniform(0.3, 0.7))))
        source = "host" if snps * samples < 1e7 and rng.random() < 0.3 else "resident"
        maf = rng.choice(["uniform", "uniform", "beta"])
        step = rng.randint(2, 5) if source == "resident" and rng.random() < 0.2 else 1
        offset = rng.randrange(step)
        missing = rng.choice([0.002, 0.01, 0.03]) if order < 4 and step == 1 and rng.random() < 0.1 else 0.0
        c = _scan("", order, snps, cases, samples - cases, _log(rng, 5, 1000), source, maf, step, offset, missing)
        del c["name"]
        most = _MISSING_WORK if missing else _MOST_WORK[order]
        if _combos(c) <= _MOST_COMBOS[order] and _combos(c) * samples <= most:
            return c


def _parts(case):
    """The scans of a case (a batch's follow from its `base`)."""
    if "scans" not in case:
        return [case]
    out = []
    for i in range(case["scans"]):
        rng = np.random.default_rng(case["base"] + i)
        order = 2 + i % 3
        hi = case["order4_cap"] if order == 4 else case["max_snps"]
        snps = int(round(math.exp(rng.uniform(math.log(min(200, hi // 2)), math.log(hi)))))
        samples = int(round(math.exp(rng.uniform(math.log(case["min_samples"]), math.log(case["max_samples"])))))
        cases = int(round(samples * rng.uniform(0.3, 0.7)))
        out.append(_scan("", order, snps, cases, samples - cases, case["outputs"]))
    return out


def _genotypes(c, seed):
    """(codes uint8 [snps, samples] on the GPU, cases first; 3 where a call is missing)."""
    n, m = c["snps"], c["cases"] + c["ctrls"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    maf = torch.empty(n, device="cuda")
    if c["maf"] == "uniform":
        maf.uniform_(0.05, 0.5, generator=g)
    else:  # Beta(1/2, 1/2) on [0.01, 0.5]: the arcsine law, by its inverse
        u = torch.rand(n, device="cuda", generator=g)
        lo = math.asin(math.sqrt(0.01))
        maf = torch.sin(lo + u * (math.asin(math.sqrt(0.5)) - lo)) ** 2
    q0, q2 = ((1 - maf) ** 2)[:, None], (1 - maf * maf)[:, None]

    def hwe(u, r):
        return (u >= q0[r]).to(torch.uint8) + (u >= q2[r]).to(torch.uint8)

    codes = torch.empty(n, m, dtype=torch.uint8, device="cuda")
    for s in range(0, n, 4096):
        r = slice(s, min(n, s + 4096))
        codes[r] = hwe(torch.rand(r.stop - r.start, m, device="cuda", generator=g), r)
    # the planted interaction: individuals who carry a minor allele at each of `order` SNPs are cases
    # with probability 0.65; individuals are drawn until both classes are full
    rows = torch.randperm(n, device="cuda", generator=g)[:c["order"]]
    pool = hwe(torch.rand(c["order"], 8 * m, device="cuda", generator=g), rows)
    p = torch.where((pool >= 1).all(0), 0.65, 0.5)
    is_case = torch.rand(8 * m, device="cuda", generator=g) < p
    pick = torch.cat([is_case.nonzero()[:c["cases"], 0], (~is_case).nonzero()[:c["ctrls"], 0]])
    codes[rows] = pool[:, pick]
    if c["missing"]:
        for s in range(0, n, 4096):
            r = slice(s, min(n, s + 4096))
            codes[r][torch.rand(r.stop - r.start, m, device="cuda", generator=g) < c["missing"]] = 3
    return codes


def _seeds(case, seed):
    return [seed * 1000003 + 7919 * i + 1 for i in range(len(_parts(case)))]


def prepare(case, seed):
    gs = GpuSearch(0)
    scans = []
    for c, s in zip(_parts(case), _seeds(case, seed)):
        codes = _genotypes(c, s).cpu().numpy()
        is_case = np.arange(codes.shape[1]) < c["cases"]
        if c["source"] == "host":
            data = Dataset.from_genotypes(codes, is_case)
        else:
            data = upload_genotypes(gs.ctx, codes, is_case)
        scans.append((data, c["order"], Distribution(c["snps"], c["order"] - 1, c["step"], c["offset"]), c["outputs"]))
    return {"search": gs, "scans": scans, "batch": "scans" in case}


def _arrays(results, order):
    return [np.array([r.combination for r in results], np.int32).reshape(-1, order),
            np.array([r.val for r in results], np.float32)]


def run(state):
    gs, scans = state["search"], state["scans"]
    if state["batch"]:
        out = []
        for (results, mi), s in zip(gs.run_batch(scans), scans):
            out += _arrays(results, s[1]) + [mi]
        return out
    data, order, dist, outputs = scans[0]
    return _arrays(gs.run(data, order, dist, outputs), order)


def work(case):
    b = f = 0.0
    for c in _parts(case):
        b += 3 * c["snps"] * (c["cases"] + c["ctrls"]) / 8 + c["outputs"] * (4 * c["order"] + 4)
        f += _flops(c) if not c["missing"] else 2.0 * 3 ** c["order"] * _combos(c) * (c["cases"] + c["ctrls"])
    return {"bytes": b, "flops": f}


def _xlogx(t):
    return torch.special.xlogy(t, t)


def _exact_scan(c, codes):
    """The best MI values of a scan in 64 bits, best first: every combination's table by matrix products of
    genotype indicators (whole numbers, exact in FP32 with its own 24 bits), the entropies in FP64."""
    n, k, n1, n0 = c["snps"], c["order"], c["cases"], c["ctrls"]
    N = n1 + n0
    one = torch.stack([codes == g for g in range(3)], 1).float()  # [snps, 3, samples]
    flat = one.reshape(3 * n, N)
    h = math.log(N) - (n1 * math.log(n1) + n0 * math.log(n0)) / N
    total = math.comb(n, k - 1)
    prefixes = np.fromiter(itertools.chain.from_iterable(itertools.combinations(range(n), k - 1)), np.int32,
                           total * (k - 1)).reshape(total, k - 1)[c["offset"]::c["step"]]
    prefixes = torch.from_numpy(prefixes).long().cuda()
    rows = 3 ** (k - 1)
    chunk = max(1, int(6e8 / (rows * (3 * n + N))))
    best = torch.empty(0, dtype=torch.float64, device="cuda")
    for s in range(0, len(prefixes), chunk):
        p = prefixes[s:s + chunk]
        first = int(p[:, -1].min()) + 1
        if first >= n:
            continue
        a = one[p[:, 0]]
        for t in range(1, k - 1):
            a = (a[:, :, None] * one[p[:, t]][:, None]).reshape(len(p), -1, N)
        a = a.reshape(-1, N)
        tab = [(a[:, r] @ flat[3 * first:, r].T).reshape(len(p), rows, n - first, 3)
               for r in (slice(0, n1), slice(n1, N))]
        mi = torch.zeros(len(p), n - first, dtype=torch.float64, device="cuda")
        for g in range(rows):
            x, y = tab[0][:, g].double(), tab[1][:, g].double()
            mi += (_xlogx(x) + _xlogx(y) - _xlogx(x + y)).sum(-1)
        mi = mi / N + h
        mi[torch.arange(first, n, device="cuda")[None] <= p[:, -1:]] = -1.0
        best = torch.cat([best, mi.flatten()])
        best = best.topk(min(c["outputs"], len(best))).values
    return best[best >= -0.5].cpu().numpy()


def exact(case, seed):
    parts = _parts(case)
    # about 20 s of FP64 logarithms and FP32 products
    if sum(_combos(c) * 3 ** c["order"] for c in parts) > 2.5e9 or \
            sum(_combos(c) * 3 ** c["order"] * (c["cases"] + c["ctrls"]) for c in parts) > 4e13:
        return None
    out = []
    for c, s in zip(parts, _seeds(case, seed)):
        mi = _exact_scan(c, _genotypes(c, s))
        out += [None, mi] + ([mi] if "scans" in case else [])
    return out
