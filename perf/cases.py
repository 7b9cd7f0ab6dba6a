"""The calls that are timed: what a program does with this package, over the range it does it in.

A case is a cohort (samples x sites) or a few of them, the estimator run on it and the options given.  Sizes and
distributions follow kestrel_b200/synth.py and bench.py: REF frequencies Beta(1/2, 1/2) within [0.05, 0.95],
Hardy-Weinberg genotypes, independent missing calls, some first-degree relatives and inbred samples.  Every pass takes
new host arrays through the whole public call (upload, frequencies, all pairs, rows back), with one Estimator per
process and precision, as a program that estimates cohort after cohort keeps it; a serving panel is loaded before.

Outputs are, per pair, the Jacquard coefficients as far as two-allele sites determine them (see determined()), the
kinship and the objective, in the type of the arithmetic that the caller chose: precision "fp32c" (the default)
evaluates sites in FP32, so its rows hold about seven digits in their doubles and are kept as float32, as a program
that stores them would; precision "fp64" stays float64.  The rows' iteration counts and condition estimates say how
the solver went and are not kept.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from kestrel_b200 import KINSHIP_VECTOR, OUTPUT_DTYPE, Estimator

EPS = 1e-8   # the estimator's epsilon inside the logarithm
# exact() enumerates every pair-site: above this many it is left out
EXACT_PAIR_SITES = 7e8


def listed():
    return [
        # a nuclear family or a few candidate duplicates on a small panel: latency
        {"name": "ml_family_6x1500", "kind": "ml", "n": 6, "m": 1500, "missing": 0.02, "related": 0.6, "inbred": 0.0, "af": False, "precision": "fp32c"},
        # the CPU-sized cohort of the configurations (64 x 10,000, 2% missing)
        {"name": "ml_64x10000", "kind": "ml", "n": 64, "m": 10000, "missing": 0.02, "related": 0.0, "inbred": 0.0, "af": False, "precision": "fp32c"},
        # an ordinary cohort, odd sizes, uneven missingness, inbred samples, the caller's frequencies
        {"name": "ml_201x33333_af", "kind": "ml", "n": 201, "m": 33333, "missing": 0.1, "related": 0.3, "inbred": 0.25, "af": True, "precision": "fp32c"},
        # the benchmark's cohort
        {"name": "ml_1024x100000", "kind": "ml", "n": 1024, "m": 100000, "missing": 0.02, "related": 0.5, "inbred": 0.0, "af": False, "precision": "fp32c"},
        # the FP64 form, asked for where the rows are compared or differenced
        {"name": "ml_fp64_96x20000", "kind": "ml", "n": 96, "m": 20000, "missing": 0.05, "related": 0.3, "inbred": 0.1, "af": False, "precision": "fp64"},
        # the default hard-call estimator of the CLI (conditional least squares): small and large
        {"name": "cls_64x10000", "kind": "cls", "n": 64, "m": 10000, "missing": 0.0, "related": 0.2, "inbred": 0.0, "af": False, "precision": "fp32c"},
        {"name": "cls_1024x100000", "kind": "cls", "n": 1024, "m": 100000, "missing": 0.0, "related": 0.2, "inbred": 0.0, "af": False, "precision": "fp32c"},
        # genotype likelihoods of low-coverage data
        {"name": "soft_200x15000", "kind": "soft", "n": 200, "m": 15000, "missing": 0.02, "related": 0.2, "inbred": 0.0, "af": False, "precision": "fp32c"},
        # several cohorts in one call, uneven, one missing rate per sample
        {"name": "batch_4_cohorts", "kind": "batch", "n": 384, "m": 65000, "missing": 0.1, "related": 0.2, "inbred": 0.1, "af": False, "precision": "fp32c", "cohorts": 4},
        # a few query samples against a resident panel, some of the panel's sites called
        {"name": "serve_12_on_512x20000", "kind": "serve", "n": 512, "m": 20000, "missing": 0.02, "related": 0.0, "inbred": 0.0, "af": False, "precision": "fp32c", "queries": 12},
    ]


def draw(rng):
    """A case of the same ranges: 2 to 1,024 samples, 500 to 100,000 sites."""
    kind = rng.choice(["ml", "ml", "ml", "cls", "soft", "batch", "serve"])
    precision = "fp64" if kind == "ml" and rng.random() < 0.25 else "fp32c"
    top = {"ml": 1024, "cls": 1024, "soft": 256, "batch": 512, "serve": 1024}[kind]
    most = {"ml": 2e10, "cls": 2e10, "soft": 4e8, "batch": 4e9, "serve": 4e8}[kind] / (20 if precision == "fp64" else 1)
    for _ in range(1000):
        n = round(math.exp(rng.uniform(math.log(2), math.log(top))))
        m = round(math.exp(rng.uniform(math.log(500), math.log(100000))))
        queries = rng.randint(1, 64) if kind == "serve" else 0
        pairs = n * queries if kind == "serve" else n * (n + 1) / 2
        if pairs * m <= most and (kind != "serve" or n >= 32):
            break
    case = {"kind": kind, "n": n, "m": m, "missing": 0.0 if kind == "cls" else round(rng.uniform(0.0, 0.2), 3),
            "related": round(rng.uniform(0.0, 0.6), 2), "inbred": round(rng.uniform(0.0, 0.3), 2) if kind != "cls" else 0.0,
            "af": kind == "ml" and rng.random() < 0.3, "precision": precision}
    if kind == "serve":
        case["queries"] = queries
    if kind == "batch":
        case["cohorts"] = rng.randint(2, 6)
    return case


# ------------------------------------------------------------------ inputs

def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def cohort(n, m, missing, related, inbred, gen):
    """(codes u8 [n, m] on the device, 3 = missing; REF frequencies [m])."""
    dev = gen.device
    rand = lambda *s: torch.rand(*s, generator=gen, device=dev)  # noqa: E731
    p = torch.sin(0.5 * math.pi * rand(m)).square().clamp(0.05, 0.95).double()
    q = (1.0 - p).float()
    a1 = (rand(n, m) < q).to(torch.uint8)
    a2 = (rand(n, m) < q).to(torch.uint8)
    # first- and second-degree relatives: sample 2k + 1 shares alleles of sample 2k by descent
    for k in range(int(related * n / 2)):
        one, both = [(1.0, 0.0), (0.5, 0.25), (0.5, 0.0)][k % 3]   # parent-offspring, full, half sibs
        u = rand(m)
        a1[2 * k + 1] = torch.where(u < one + both, a1[2 * k], a1[2 * k + 1])
        a2[2 * k + 1] = torch.where(u < both, a2[2 * k], a2[2 * k + 1])
    for s in range(n - int(inbred * n), n):
        f = 0.0625 + 0.1875 * ((s * 7) % 5) / 4.0
        a2[s] = torch.where(rand(m) < f, a1[s], a2[s])
    codes = a1 + a2
    if missing > 0:
        rate = 2.0 * missing * rand(n, 1) if missing >= 0.05 else torch.full((n, 1), missing, device=dev)
        codes[rand(n, m) < rate] = 3
    return codes, p


def generator(seed):
    g = torch.Generator(device=device())
    g.manual_seed(seed)
    return g


def to_host(t):
    """A host array as a program that uploads much keeps it: page-locked."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    h.copy_(t)
    return h.numpy()


def rows_buffer(pairs):
    h = torch.zeros(max(pairs, 1) * 14, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return h.numpy().view(OUTPUT_DTYPE)


def batch_sizes(case):
    """Uneven cohorts: samples and sites fall by a third from one to the next."""
    return [(max(2, round(case["n"] / 1.5 ** k)), max(200, round(case["m"] / 1.25 ** k))) for k in range(case["cohorts"])]


def likelihoods(codes, gen):
    """Linear-scale genotype likelihoods [n, m, 3] around the calls: 0 to 20 percent off the call, NaN where missing."""
    n, m = codes.shape
    off = 0.2 * torch.rand(n, m, 1, generator=gen, device=gen.device).double().square()
    mix = torch.rand(n, m, 3, generator=gen, device=gen.device).double()
    gl = off * mix
    c = codes.long().clamp(max=2).unsqueeze(2)
    gl.scatter_(2, c, 1.0)
    gl[codes == 3] = float("nan")
    return gl


def inputs(case, seed):
    """The case's arrays on the device, made from the seed alone."""
    gen = generator(seed)
    args = (case["missing"], case["related"], case["inbred"], gen)
    if case["kind"] == "batch":
        return {"cohorts": [cohort(n, m, *args) for n, m in batch_sizes(case)]}
    codes, p = cohort(case["n"], case["m"], *args)
    d = {"codes": codes, "p": p}
    if case["kind"] == "soft":
        d["gl"] = likelihoods(codes, gen)
    if case["kind"] == "serve":
        nq = case["queries"]
        q = (1.0 - p).float()
        a = torch.rand(2, nq, case["m"], generator=gen, device=gen.device) < q
        d["query"] = a[0].to(torch.uint8) + a[1].to(torch.uint8)
        d["query"][torch.rand(nq, case["m"], generator=gen, device=gen.device) < 0.02] = 3
        d["mask"] = (torch.rand(case["m"], generator=gen, device=gen.device) < 0.8).to(torch.uint8)
    return d


_kept = {}


def estimator(precision):
    if precision not in _kept:
        _kept[precision] = Estimator(precision=precision)
    return _kept[precision]


def prepare(case, seed):
    d = inputs(case, seed)
    n, kind = case["n"], case["kind"]
    s = {"case": case, "pairs": n * (n + 1) // 2}
    if kind == "batch":
        s["cohorts"] = [(to_host(c), None, None) for c, _ in d["cohorts"]]
        s["out"] = [rows_buffer(c.shape[0] * (c.shape[0] + 1) // 2) for c, _ in d["cohorts"]]
        s["est"] = estimator(case["precision"])
        return s
    if kind == "serve":
        s["est"] = Estimator(precision=case["precision"])
        s["est"].panel_load(to_host(d["codes"]))
        s["query"], s["mask"] = to_host(d["query"]), to_host(d["mask"])
        return s
    s["est"] = estimator(case["precision"])
    s["out"] = rows_buffer(s["pairs"])
    if kind == "soft":
        s["gl"] = to_host(d["gl"])
    else:
        s["codes"] = to_host(d["codes"])
        s["af"] = np.ascontiguousarray(torch.stack([d["p"], 1.0 - d["p"]], 1).cpu().numpy()) if case["af"] else None
    return s


def determined(like):
    """The projection of the coefficients onto what two-allele sites determine.  At every such site the likelihood is the
    same all along (0, 1, 0, -1, 0, -1, -1, 2, 0): where an optimum can move along it (1% of the pairs of an outbred
    cohort, 5% of an inbred one), its place there is no estimate, and the two precisions differ in it by 0.01 to 0.03."""
    v = torch.tensor([0.0, 1, 0, -1, 0, -1, -1, 2, 0], dtype=torch.float64, device=like.device)
    return (torch.eye(9, dtype=torch.float64, device=like.device) - torch.outer(v, v) / (v @ v)).to(like.dtype)


def result(t):
    """[pairs, 10] coefficients and objective as the program keeps them."""
    d = t[:, :9]
    return {"delta": d @ determined(d), "kinship": d @ torch.from_numpy(KINSHIP_VECTOR).to(d), "objective": t[:, 9]}


def values(rows, precision):
    """The rows in the precision that they were estimated in."""
    t = torch.from_numpy(rows.view(np.float64).reshape(-1, 14))[:, 2:12]
    return result(t.clone() if precision == "fp64" else t.float())


def run(state):
    case, est = state["case"], state["est"]
    kind, precision = case["kind"], case["precision"]
    if kind == "batch":
        rows = est.relatedness_batch(state["cohorts"], out=state["out"])
        return [values(r, precision) for r in rows]
    if kind == "serve":
        return values(est.wait(est.submit(state["query"], state["mask"])), precision)
    if kind == "soft":
        return values(est.load_likelihoods(state["gl"]).relatedness_gl(out=state["out"]), precision)
    est.load(state["codes"], state["af"])
    rows = est.relatedness_gt(out=state["out"]) if kind == "cls" else est.relatedness(out=state["out"])
    return values(rows, precision)


def work(case):
    """Inputs read once, rows written once; per pair-site one evaluation of its nine-term mixture (18 operations)."""
    if case["kind"] == "batch":
        sizes = batch_sizes(case)
        pairs = [n * (n + 1) // 2 for n, _ in sizes]
        return {"bytes": sum(n * m for n, m in sizes) + 40 * sum(pairs), "flops": 18 * sum(k * m for k, (_, m) in zip(pairs, sizes))}
    n, m = case["n"], case["m"]
    pairs = n * case["queries"] if case["kind"] == "serve" else n * (n + 1) // 2
    read = {"soft": 24 * n * m, "serve": case.get("queries", 0) * m + n * m}.get(case["kind"], n * m)
    return {"bytes": read + (80 if case["precision"] == "fp64" else 40) * pairs, "flops": 18 * pairs * m}


# ------------------------------------------------------------ in 64 bits

def rows_table(p):
    """m[site, gx, gy, 9] in 64 bits: the probability of the joint genotype given each Jacquard state, by the states'
    identity classes over every ordering of the two genotypes' alleles."""
    classes = [(0, 0, 0, 0), (0, 0, 1, 1), (0, 0, 0, 1), (0, 0, 1, 2), (0, 1, 0, 0), (0, 1, 2, 2), (0, 1, 0, 1), (0, 1, 0, 2), (0, 1, 2, 3)]
    f = torch.stack([p, 1.0 - p])
    orders = {0: [(0, 0)], 1: [(0, 1), (1, 0)], 2: [(1, 1)]}
    out = torch.zeros(p.numel(), 3, 3, 9, dtype=torch.float64, device=p.device)
    for gx in range(3):
        for gy in range(3):
            for k, cl in enumerate(classes):
                for x in orders[gx]:
                    for y in orders[gy]:
                        al, who = x + y, {}
                        if all(who.setdefault(c, a) == a for c, a in zip(cl, al)):
                            t = torch.ones_like(p)
                            for a in who.values():
                                t = t * f[a]
                            out[:, gx, gy, k] += t
    return out


def fit_frequencies(gl, maf=None):
    """Per site the maximiser p of sum log(eps + p^2 l0 + 2 p q l1 + q^2 l2) over the called samples, with the default
    minor-allele cut 1 / (2 n); (p, kept)."""
    n = gl.shape[0]
    l = torch.nan_to_num(gl)
    called = ~torch.isnan(gl).any(2)
    w = called.double()
    p = ((2 * l[..., 0] + l[..., 1]) / l.sum(2).clamp(min=1e-300) * w).sum(0) / (2 * w.sum(0)).clamp(min=1.0)
    p = p.clamp(1e-7, 1 - 1e-7)
    for _ in range(60):
        q = 1.0 - p
        d = EPS + p * p * l[..., 0] + 2 * p * q * l[..., 1] + q * q * l[..., 2]
        d1 = 2 * p * l[..., 0] + 2 * (q - p) * l[..., 1] - 2 * q * l[..., 2]
        d2 = 2 * l[..., 0] - 4 * l[..., 1] + 2 * l[..., 2]
        f1 = (w * d1 / d).sum(0)
        f2 = (w * (d2 / d - (d1 / d) ** 2)).sum(0)
        step = torch.where(f2 < 0, -f1 / f2, 0.1 * torch.sign(f1) * torch.minimum(p, q))
        p = torch.minimum(torch.maximum(p + step, 0.25 * p), 1 - 0.25 * q).clamp(1e-9, 1 - 1e-9)
    cut = 1.0 / (2.0 * n)
    return p, (w.sum(0) > 0) & (p >= cut) & (1.0 - p >= cut)


def mixture_optimum(L):
    """Per pair the minimiser x on the simplex of -(1/n) sum log(eps + L x) and its value, by a primal-dual interior
    point method and Newton steps on the free coordinates.  L: [pairs, sites, 9], NaN rows left out."""
    ok = ~torch.isnan(L[..., 0])
    L = torch.nan_to_num(L)
    n = ok.sum(1).double()
    P, dev = L.shape[0], L.device

    def grad_hess(x):
        d = EPS + torch.bmm(L, x.unsqueeze(2)).squeeze(2)
        b = L * (ok / d).unsqueeze(2)
        g = -b.sum(1) / n[:, None]
        return g, torch.bmm(b.transpose(1, 2), b) / n[:, None, None], -(torch.log(d) * ok).sum(1) / n

    x = torch.full((P, 9), 1.0 / 9, dtype=torch.float64, device=dev)
    lam = torch.ones_like(x)
    nu = torch.zeros(P, dtype=torch.float64, device=dev)
    K = torch.zeros(P, 10, 10, dtype=torch.float64, device=dev)
    for it in range(48):
        g, H, _ = grad_hess(x)
        mu = (0.1 * (x * lam).mean(1, keepdim=True)).clamp(min=1e-14)
        K[:, :9, :9] = H + torch.diag_embed(lam / x)
        K[:, :9, 9] = -1.0
        K[:, 9, :9] = 1.0
        rhs = torch.cat([-(g - nu[:, None] - mu / x), 1.0 - x.sum(1, keepdim=True)], 1)
        s = torch.linalg.solve(K, rhs.unsqueeze(2)).squeeze(2)
        dx = s[:, :9]
        dl = mu / x - lam - lam / x * dx
        far = lambda v, dv: (0.95 / (-dv / v).clamp(min=0.95).amax(1)).clamp(max=1.0)[:, None]  # noqa: E731
        t = far(x, dx)
        for _ in range(8):   # a shorter step where the objective with the barrier would not go down
            v0, v1 = grad_hess(x)[2] - (mu * torch.log(x)).sum(1), grad_hess(x + t * dx)[2] - (mu * torch.log(x + t * dx)).sum(1)
            up = v1 > v0 + 1e-12
            if not bool(up.any()):
                break
            t = torch.where(up[:, None], 0.5 * t, t)
        x = x + t * dx
        lam = lam + far(lam, dl) * dl
        nu = nu + s[:, 9]
    free = x > lam
    x = torch.where(free, x, torch.zeros_like(x))
    x = x / x.sum(1, keepdim=True)
    for it in range(8):
        g, H, _ = grad_hess(x)
        at = (x * g).sum(1, keepdim=True)
        free = (x > 0) | (g < at - 1e-11)
        m = free.double()
        K.zero_()
        K[:, :9, :9] = H * m[:, :, None] * m[:, None, :] + torch.diag_embed(1.0 - m)
        K[:, :9, 9] = -m
        K[:, 9, :9] = m
        rhs = torch.cat([-g * m, torch.zeros(P, 1, dtype=torch.float64, device=dev)], 1)
        s = torch.linalg.solve(K, rhs.unsqueeze(2)).squeeze(2)[:, :9]
        far = 1.0 / torch.where(s < 0, -s / x.clamp(min=1e-300), torch.zeros_like(s)).amax(1, keepdim=True).clamp(min=1.0)
        x = (x + far * s).clamp(min=0.0)
        x = torch.where(x < 1e-13, torch.zeros_like(x), x)
        x = x / x.sum(1, keepdim=True)
    return x, grad_hess(x)[2]


def optimum_rows(like_x, like_y, p, pairs):
    """[pairs, 10]: the optimum and its objective for each (x, y); like_*: likelihoods [samples, sites, 3]."""
    table = rows_table(p)
    out = []
    step = max(1, (1 << 24) // p.numel())
    for at in range(0, len(pairs[0]), step):
        x, y = pairs[0][at: at + step], pairs[1][at: at + step]
        L = torch.zeros(len(x), p.numel(), 9, dtype=torch.float64, device=p.device)
        for gx in range(3):
            for gy in range(3):
                L += (like_x[x, :, gx] * like_y[y, :, gy]).unsqueeze(2) * table[:, gx, gy]
        d, f = mixture_optimum(L)
        out.append(torch.cat([d, f[:, None]], 1))
    return torch.cat(out)


def one_hot(codes):
    gl = torch.zeros(*codes.shape, 3, dtype=torch.float64, device=codes.device)
    gl.scatter_(2, codes.long().clamp(max=2).unsqueeze(2), 1.0)
    gl[codes == 3] = float("nan")
    return gl


def triangle(n, dev):
    i = torch.triu_indices(n, n, device=dev)
    return i[0], i[1]


def least_squares_rows(codes):
    """[pairs, 10]: the minimiser on the simplex of D'QD / 2 + c'D of conditional least squares over the sites that
    every sample calls, frequencies by counts, and the Brier score; a self pair on states 1 and 7.  The support is
    found among all of them."""
    codes = codes[:, (codes < 3).all(0)]
    n, m = codes.shape
    dev = codes.device
    p = 1.0 - codes.double().mean(0) / 2
    table = rows_table(p)
    Q = torch.einsum("sabi,sabj->ij", table, table) / m
    X = [(codes == g).double() for g in range(3)]
    C = torch.zeros(n, n, 9, dtype=torch.float64, device=dev)
    for gx in range(3):
        for gy in range(3):
            for k in range(9):
                C[..., k] += (X[gx] * table[:, gx, gy, k]) @ X[gy].T
    x, y = triangle(n, dev)
    c = -C[x, y] / m

    def best_of(supports):
        best = torch.full((len(x),), float("inf"), dtype=torch.float64, device=dev)
        arg = torch.zeros(len(x), 9, dtype=torch.float64, device=dev)
        for s in supports:
            s = torch.tensor(s, device=dev)
            k = len(s)
            K = torch.zeros(k + 1, k + 1, dtype=torch.float64, device=dev)
            K[:k, :k] = Q[s][:, s]
            K[:k, k] = K[k, :k] = 1.0
            inv, info = torch.linalg.inv_ex(K)
            if int(info):
                continue
            b = torch.cat([-c[:, s], torch.ones(len(x), 1, dtype=torch.float64, device=dev)], 1)
            z = (b @ inv.T)[:, :k]
            v = 0.5 * ((z @ Q[s][:, s]) * z).sum(1) + (c[:, s] * z).sum(1)
            take = (z.amin(1) >= -1e-13) & (v < best)
            best = torch.where(take, v, best)
            full = torch.zeros_like(arg)
            full[:, s] = z
            arg = torch.where(take[:, None], full, arg)
        return arg

    d = best_of([[i for i in range(9) if b >> i & 1] for b in range(1, 512)])
    d = torch.where((x == y)[:, None], best_of([[0], [6], [0, 6]]), d)
    brier = ((d @ Q) * d).sum(1) + 2 * (c * d).sum(1) + 1.0
    return torch.cat([d, brier[:, None]], 1)


def exact(case, seed):
    w = work(case)
    limit = 3e9 if case["kind"] == "cls" else EXACT_PAIR_SITES
    if w["flops"] / 18 > limit:
        return None
    d = inputs(case, seed)
    with torch.no_grad():
        if case["kind"] == "cls":
            return result(least_squares_rows(d["codes"]))
        if case["kind"] == "batch":
            got = []
            for codes, _ in d["cohorts"]:
                gl = one_hot(codes)
                p, kept = fit_frequencies(gl)
                gl = gl[:, kept].contiguous()
                got.append(result(optimum_rows(gl, gl, p[kept], triangle(len(gl), gl.device))))
            return got
        gl = d["gl"] if case["kind"] == "soft" else one_hot(d["codes"])
        p, kept = (d["p"], torch.ones_like(d["p"], dtype=torch.bool)) if case["af"] else fit_frequencies(gl)
        if case["kind"] == "serve":
            q = torch.where(d["mask"].bool()[None], d["query"], torch.full_like(d["query"], 3))
            nq, n = case["queries"], case["n"]
            i = torch.arange(nq * n, device=gl.device)
            return result(optimum_rows(one_hot(q)[:, kept].contiguous(), gl[:, kept].contiguous(), p[kept], (i // n, i % n)))
        gl = gl[:, kept].contiguous()
        return result(optimum_rows(gl, gl, p[kept], triangle(len(gl), gl.device)))
