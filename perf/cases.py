"""The work whose speed matters to a user of this framework, as cases that a timer can run.

A case is one call, through the public entry points, of the longitudinal mixed-model
solve: a GRM product, a mixed-model solve, a block PCG, an AIREML evaluation or a whole
AIREML run, the GRM build and the loading of genotypes -- on genotypes or on a dense GRM,
in FP64 (the default of the programs and of the API) or in mixed precision.  Sizes are
those of the repository's own configurations (bench.py), of its tests, or odd ones between
them.  Inputs are made on the GPU from the seed alone.
"""
import math

import numpy as np
import torch

import globe_gb300 as G

VC = (0.6, 0.4, 0.4, 0.2, 0.2)          # sig2e, sig2g, sig2b0, sigb01, sig2b1 of the simulated cohorts
THETA0 = (0.5, 0.3, 0.2, 0.1, 0.1)      # where runAIREML starts by default
TOL = 1e-10                             # --pcgTol of a solve whose digits count: at the default 1e-5 the
                                        # solution is defined to that tolerance only, whatever the precision
MIN_MAF, MAX_MISS = 0.01, 0.2           # the programs' SNP filter
SOLVE_ITERS = 17                        # iterations that work() counts for a solve to TOL (they take 15 to 30)
DEV = "cuda"


def listed():
    return [
        # one product on a small cohort through the host interface (u-hat, checks in a script): latency
        dict(name="apply-600", kind="apply", prec="fp64", N=601, M=1503, k=1),
        # runPCGsolver --geno on the 2,000-individual configuration, in its default FP64
        dict(name="mme-2k", kind="mme", prec="fp64", N=2000, M=10000, k=5, recs="uniform", a=3, b=10),
        # the same cohort's block solve in mixed precision on device buffers: launches and latency
        dict(name="pcg-2k-mixed", kind="pcg", prec="mixed", N=2000, M=10000, k=5, recs="uniform", a=3, b=10),
        # a cohort of ordinary size in the default FP64, individuals with 1 to 200 records
        dict(name="pcg-20k", kind="pcg", prec="fp64", N=20000, M=20000, k=5, recs="geometric", a=0.1, b=200),
        # bench.py's headline workload: 12.5 GB of packed genotypes, [X y] as right-hand sides
        dict(name="pcg-100k-mixed", kind="pcg", prec="mixed", N=100000, M=500000, k=5, recs="poisson", a=6, b=0),
        # y and 64 probes as one block of 65 right-hand sides, ragged sizes
        dict(name="pcg-65rhs-mixed", kind="pcg", prec="mixed", N=100003, M=75001, k=65, recs="fixed", a=6, b=0),
        # one AIREML iteration's score and AI matrix at the biobank's record counts, 32 probes
        dict(name="eval-100k-mixed", kind="eval", prec="mixed", N=100000, M=100000, k=5, mc=32, recs="geometric", a=0.1,
             b=200),
        # a whole runAIREML on genotypes, 15 probes
        dict(name="aireml-20k-mixed", kind="aireml", prec="mixed", N=20000, M=20000, k=5, mc=15, recs="poisson", a=6, b=0),
        # the dense-GRM configuration: 16 right-hand sides
        dict(name="dense-20k-mixed", kind="dense", prec="mixed", N=20000, M=2000, k=16, recs="poisson", a=5, b=0),
        # a dense GRM of odd size in the default FP64
        dict(name="dense-6k", kind="dense", prec="fp64", N=6007, M=2000, k=5, recs="poisson", a=5, b=0),
        # buildGRM, the .grm.bin payload from genotypes
        dict(name="build-10k-mixed", kind="build", prec="mixed", N=10007, M=30011, k=1),
        # what every program does before its first solve: filter and lay out the genotypes, A_ii
        dict(name="load-100k", kind="load", prec="fp64", N=100000, M=200000, k=1),
    ]


# individuals, SNPs, individuals x SNPs: the ranges of each kind and precision that draw() spans
RANGES = {
    ("apply", "fp64"): (300, 20000, 500, 40000, 4e8), ("apply", "mixed"): (300, 60000, 500, 200000, 4e9),
    ("mme", "fp64"): (300, 20000, 500, 40000, 4e8), ("mme", "mixed"): (300, 60000, 500, 200000, 4e9),
    ("pcg", "fp64"): (300, 20000, 500, 40000, 4e8), ("pcg", "mixed"): (300, 120000, 500, 300000, 1e10),
    ("eval", "mixed"): (1000, 60000, 2000, 100000, 3e9), ("eval", "fp64"): (500, 5000, 1000, 10000, 2e7),
    ("dense", "fp64"): (300, 8000, 1000, 2000, 1e9), ("dense", "mixed"): (300, 20000, 1000, 2000, 1e9),
    ("build", "mixed"): (300, 10000, 500, 40000, 3e8), ("build", "fp64"): (300, 3000, 500, 5000, 1e7),
    ("load", "fp64"): (300, 120000, 500, 300000, 2e10),
}


def draw(rng):
    kind, prec = rng.choice(sorted(RANGES))
    n0, n1, m0, m1, most = RANGES[kind, prec]
    while True:
        N = int(round(math.exp(rng.uniform(math.log(n0), math.log(n1)))))
        M = int(round(math.exp(rng.uniform(math.log(m0), math.log(m1)))))
        if N * M <= most:
            break
    c = dict(kind=kind, prec=prec, N=N, M=M, k=1)
    if kind == "apply":
        c["k"] = rng.choice([1, 1, 3, 5, 16])
    if kind in ("mme", "pcg", "eval", "dense"):
        c["k"] = 5 if kind in ("mme", "eval") else rng.choice([5, 5, 5, 8, 16, 20, 33]) if prec == "mixed" else rng.choice([5, 8])
        c["recs"], c["a"], c["b"] = rng.choice([("uniform", 3, 10), ("poisson", 6, 0), ("poisson", 5, 0), ("fixed", 6, 0),
                                                ("geometric", 0.1, 200)])
    if kind == "eval":
        c["mc"] = rng.choice([5, 15, 32])
    return c


# ---- inputs ------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _bed(case, seed):
    """Packed PLINK rows (M x stride uint8, stride a multiple of 16): MAF U(0.01, 0.5), the counted
    allele flipped for half the SNPs, 2% missing."""
    N, M = case["N"], case["M"]
    bps, miss = (N + 3) // 4, 0.02
    out = torch.zeros((M, (bps + 15) // 16 * 16), dtype=torch.uint8, device=DEV)
    g = _gen(seed)
    p = torch.rand(M, device=DEV, generator=g) * 0.49 + 0.01
    p = torch.where(torch.rand(M, device=DEV, generator=g) < 0.5, p, 1 - p)
    step = max(1, (1 << 28) // (4 * bps))
    for s in range(0, M, step):
        q = p[s:s + step, None]
        u = torch.rand((q.shape[0], 4 * bps), device=DEV, generator=g)
        code = 3 - (u < (1 - miss) * (1 - (1 - q) ** 2)).to(torch.uint8) - 2 * (u < (1 - miss) * q * q).to(torch.uint8)
        code[u >= 1 - miss] = 1
        code[:, N:] = 0
        c = code.view(-1, bps, 4)
        out[s:s + step, :bps] = c[:, :, 0] | (c[:, :, 1] << 2) | (c[:, :, 2] << 4) | (c[:, :, 3] << 6)
    return out


def _grm(case, seed):
    """A float32 GRM of the dense cases: W'W / M, W standard normal (M x N); its packed lower triangle."""
    N, M = case["N"], case["M"]
    W = torch.randn((M, N), device=DEV, generator=_gen(seed))
    W -= W.mean(1, keepdim=True)
    A = (W.T @ W) / M
    lt = torch.empty(N * (N + 1) // 2, device=DEV)
    cols = torch.arange(N, device=DEV)
    for i in range(0, N, 2048):
        rows = cols[i:i + 2048]
        lt[i * (i + 1) // 2:(i + len(rows)) * (i + len(rows) + 1) // 2] = A[rows][cols[None, :] <= rows[:, None]]
    return lt


def _counts(case, rng):
    """Records per individual: the same numbers for every seed (so the sizes are the case's), in another order."""
    N, a, b = case["N"], case["a"], case["b"]
    own = np.random.default_rng(N)
    if case["recs"] == "uniform":
        n = own.integers(a, b + 1, size=N)
    elif case["recs"] == "poisson":
        n = own.poisson(a, size=N) + 1
    elif case["recs"] == "fixed":
        n = np.full(N, a)
    else:
        n = np.clip(own.geometric(a, size=N), 1, b)
    return rng.permutation(n)


def _cohort(case, seed, u=None):
    """Record table: intercept, two covariates and time; y from the model (u: genetic values)."""
    rng = np.random.default_rng(seed)
    N = case["N"]
    n = _counts(case, rng)
    indiv = np.repeat(np.arange(N, dtype=np.int32), n)
    T = 5.0 if case["recs"] == "uniform" else 10.0
    key = np.sort(indiv + rng.random(len(indiv)) * 0.999)      # times sorted within each individual
    t = (key - indiv) * (T / 0.999)
    X = np.asfortranarray(np.column_stack([np.ones(len(t)), rng.standard_normal((len(t), 2)), t]))
    L = np.linalg.cholesky(np.array([[VC[2], VC[3]], [VC[3], VC[4]]]))
    b = rng.standard_normal((N, 2)) @ L.T
    u = rng.standard_normal(N) * math.sqrt(VC[1]) if u is None else u
    y = X @ np.array([1.0, 0.5, -0.3, 0.1]) + u[indiv] + b[indiv, 0] + b[indiv, 1] * t
    y += rng.standard_normal(len(t)) * math.sqrt(VC[0])
    return indiv, X, y


class _Zs:
    """The standardised kept genotypes in float64 by torch, chunks of SNPs at a time."""

    def __init__(self, bed, N, rows=1 << 28):
        self.bed, self.N, self.step = bed, N, max(1, rows // N)
        self.keep, self.f = [], []
        for s in range(0, bed.shape[0], self.step):
            code = self._codes(s)
            miss = (code == 1).sum(1)
            alt = 2 * (code == 0).sum(1) + (code == 2).sum(1)
            n = N - miss
            maf = torch.where(n > 0, alt.float() / (2.0 * n.float()), torch.zeros((), device=DEV))
            lo = torch.tensor(np.float32(MIN_MAF), device=DEV)
            self.keep.append((maf >= lo) & (maf <= 1.0 - lo) & (miss.float() / torch.tensor(float(N), device=DEV) <= np.float32(MAX_MISS)))
            self.f.append(torch.where(n > 0, alt.double() / (2 * n).double().clamp(min=1), torch.zeros((), device=DEV, dtype=torch.float64)))
        self.M = int(sum(int(k.sum()) for k in self.keep))

    def _codes(self, s):
        b = self.bed[s:s + self.step, :(self.N + 3) // 4]
        return torch.stack([(b >> (2 * j)) & 3 for j in range(4)], 2).view(b.shape[0], -1)[:, :self.N]

    def chunks(self):
        for i, s in enumerate(range(0, self.bed.shape[0], self.step)):
            code, f = self._codes(s)[self.keep[i]], self.f[i][self.keep[i]]
            den = 2 * f * (1 - f)
            inv = torch.where(den > 1e-12, den.rsqrt(), torch.ones_like(den))
            # codes 0, 1, 2, 3 stand for 2, missing (0), 1, 0 copies
            z = ((code == 0).to(torch.float64) * 2).add_((code == 2).to(torch.float64))
            yield z.sub_((2 * f)[:, None]).mul_(inv[:, None])

    def apply(self, Z):
        out = torch.zeros_like(Z)
        for z in self.chunks():
            out += z.T @ (z @ Z)
        return out / max(1, self.M)

    def diag(self):
        out = torch.zeros(self.N, dtype=torch.float64, device=DEV)
        for z in self.chunks():
            out += z.square_().sum(0)
        return out / max(1, self.M)

    def values(self, seed):
        """Genetic values Zs' w sqrt(sig2g / M), w standard normal."""
        u, g = torch.zeros(self.N, dtype=torch.float64, device=DEV), _gen(seed)
        for z in self.chunks():
            u += z.T @ torch.randn(z.shape[0], device=DEV, generator=g, dtype=torch.float64)
        return (u * math.sqrt(VC[1] / max(1, self.M))).cpu().numpy()


class _DenseA:
    """The dense GRM in float64 by torch."""

    def __init__(self, lt, N):
        self.A = torch.zeros((N, N), dtype=torch.float64, device=DEV)
        cols = torch.arange(N, device=DEV)
        for i in range(0, N, 2048):
            rows = cols[i:i + 2048]
            part = torch.zeros((len(rows), N), dtype=torch.float64, device=DEV)
            part[cols[None, :] <= rows[:, None]] = lt[i * (i + 1) // 2:(i + len(rows)) * (i + len(rows) + 1) // 2].double()
            self.A[i:i + 2048] = part
        self.A += torch.tril(self.A, -1).T

    def apply(self, Z):
        return self.A @ Z

    def diag(self):
        return self.A.diagonal().clone()


def _signal(case, bed, seed):
    """Genetic values for the cases whose results depend on there being a genetic signal."""
    return _Zs(bed, case["N"]).values(seed) if case["kind"] in ("mme", "aireml", "eval") else None


def _rhs(case, X, y, seed):
    """k right-hand sides, one a row (column-major): [X y], then standard normal probes."""
    B = torch.randn((case["k"], len(y)), dtype=torch.float64, device=DEV, generator=_gen(seed))
    own = torch.from_numpy(np.ascontiguousarray(np.column_stack([X, y]).T)).to(DEV)
    B[:own.shape[0]] = own[:case["k"]]
    return B


def _z(case, seed):
    return np.asfortranarray(np.random.default_rng(seed).standard_normal((case["N"], case["k"])))


def prepare(case, seed):
    """A context with the inputs loaded, the components set and, for the device entry points, the buffers."""
    kind, N = case["kind"], case["N"]
    ctx = G.Context(0)
    s = dict(case=case, ctx=ctx, prec=G.PREC_MIXED if case["prec"] == "mixed" else G.PREC_FP64)
    if kind == "dense":
        indiv, X, y = _cohort(case, seed)
        ctx.load_records(indiv, X, y, N)
        ctx.load_grm(_grm(case, seed).cpu().numpy(), N)
    else:
        bed = _bed(case, seed)
        if kind in ("build", "load"):
            ctx.set_individuals(N)
        elif kind == "apply":
            ctx.load_records(np.arange(N, dtype=np.int32), np.ones((N, 1)), np.zeros(N), N)
        else:
            indiv, X, y = _cohort(case, seed, _signal(case, bed, seed))
            ctx.load_records(indiv, X, y, N)
        if kind == "load":
            torch.cuda.synchronize()
            s["bed"] = bed
        else:
            torch.cuda.synchronize()                    # the context's stream does not wait for torch's
            ctx.load_bed_dev(bed.data_ptr(), case["M"], bed.shape[1], MIN_MAF, MAX_MISS)
    ctx.set_vc(THETA0 if kind == "eval" else VC)
    if kind in ("apply", "build"):
        ctx.set_precision(s["prec"])
    if kind == "apply":
        s["Z"] = _z(case, seed)
    if kind == "build":
        s["lt"] = torch.empty(N * (N + 1) // 2, device=DEV)
    if kind in ("pcg", "dense"):
        s["B"] = _rhs(case, X, y, seed)
        s["X"] = torch.empty_like(s["B"])
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "apply":
        return ctx.grm_apply(s["Z"])
    if kind == "mme":
        r = ctx.mme(tol=TOL, rule=G.RULE_PCGSOLVER, x0mode=G.X0_ZERO, precision=s["prec"])
        return [r["beta"], r["uhat"], r["bhat"], r["vinv_r"]]
    if kind in ("pcg", "dense"):
        ctx.pcg_dev(s["B"].data_ptr(), s["X"].data_ptr(), case["k"], tol=TOL, rule=G.RULE_PCGSOLVER, x0mode=G.X0_ZERO,
                    precision=s["prec"])
        return s["X"]
    if kind == "eval":
        r = ctx.aireml_eval(case["mc"], seed=12345, tol=TOL, precision=s["prec"])
        return [r["first"], r["trace"], r["grad"], ctx.aireml_ai(tol=TOL, precision=s["prec"])]
    if kind == "aireml":
        r = ctx.aireml_run(theta0=THETA0, numMC=case["mc"], pcg_tol=TOL, precision=s["prec"])
        return [r["theta"], r["se"], r["ai"], r["iterations"]]
    if kind == "build":
        ctx.grm_build_dev(s["lt"].data_ptr())
        return s["lt"]
    kept = ctx.load_bed_dev(s["bed"].data_ptr(), case["M"], s["bed"].shape[1], MIN_MAF, MAX_MISS)
    return [ctx.genetic_diag(), kept]


def work(case):
    """Genotypes (or the GRM) stream once per product, since a product needs the one before; the
    right-hand sides and results once."""
    N, M, k, kind = case["N"], case["M"], case["k"], case["kind"]
    geno = M * ((N + 3) // 4)
    mean = {"uniform": 6.5, "poisson": case.get("a", 0) + 1, "fixed": 6, "geometric": 10}.get(case.get("recs"), 0)
    rec = 8 * N * mean
    if kind == "apply":
        return {"bytes": geno + 16 * N * k, "flops": 4 * N * M * k}
    if kind == "dense":
        return {"bytes": SOLVE_ITERS * 2 * N * (N + 1) + 2 * rec * k, "flops": SOLVE_ITERS * 2 * N * N * k}
    if kind in ("mme", "pcg"):
        return {"bytes": SOLVE_ITERS * geno + 2 * rec * k, "flops": SOLVE_ITERS * 4 * N * M * k}
    if kind in ("eval", "aireml"):
        one = k + case["mc"]                            # one block solve of [X y | probes], one of the AI matrix
        evals = 1 if kind == "eval" else 11             # gradient evaluations of a whole run
        return {"bytes": evals * (2 * SOLVE_ITERS + 2) * geno + 6 * rec, "flops": evals * (SOLVE_ITERS + 1) * 4 * N * M * (one + 5)}
    if kind == "build":
        return {"bytes": geno + 2 * N * (N + 1), "flops": N * (N + 1) * M}
    return {"bytes": 2 * geno + 8 * N, "flops": 2 * N * M}  # the payload in, the resident copy out


# ---- the same in 64 bits, by torch --------------------------------------------

class _Model:
    def __init__(self, A, indiv, X, N, vc):
        self.A, self.N, self.vc = A, N, vc
        self.i = torch.from_numpy(indiv.astype(np.int64)).to(DEV)
        self.X = torch.from_numpy(np.ascontiguousarray(X)).to(DEV)
        self.t = self.X[:, -1:].clone()
        g = A.diag()
        n = self.sums(torch.ones_like(self.t))[:, 0]
        st, stt = self.sums(self.t)[:, 0], self.sums(self.t * self.t)[:, 0]
        e, s2g, b0, b01, b1 = vc
        C = torch.stack([torch.stack([b0 + s2g * g, torch.full_like(g, b01)], 1),
                         torch.stack([torch.full_like(g, b01), torch.full_like(g, b1)], 1)], 1)
        W = torch.stack([torch.stack([n, st], 1), torch.stack([st, stt], 1)], 1)
        self.H = torch.linalg.solve(e * torch.eye(2, dtype=torch.float64, device=DEV) + C @ W, C)

    def sums(self, x):
        return torch.zeros((self.N, x.shape[1]), dtype=torch.float64, device=DEV).index_add_(0, self.i, x)

    def V(self, x):
        e, s2g, b0, b01, b1 = self.vc
        s0, s1 = self.sums(x), self.sums(self.t * x)
        a0 = s2g * self.A.apply(s0) + b0 * s0 + b01 * s1
        return a0[self.i] + self.t * (b01 * s0 + b1 * s1)[self.i] + e * x

    def Qinv(self, r):
        s = torch.stack([self.sums(r), self.sums(self.t * r)], 1)
        g = self.H @ s
        return (r - g[:, 0][self.i] - self.t * g[:, 1][self.i]) / self.vc[0]

    def solve(self, B, tol=TOL):
        """Block PCG from 0 until max |r|/|b| < tol."""
        x, r = torch.zeros_like(B), B.clone()
        z = self.Qinv(r)
        p, rz, nb = z.clone(), (r * z).sum(0), B.norm(dim=0)
        for _ in range(200):
            q = self.V(p)
            a = rz / (p * q).sum(0)
            x += a * p
            r -= a * q
            if float((r.norm(dim=0) / nb).max()) < tol:
                break
            z = self.Qinv(r)
            new = (r * z).sum(0)
            p = z + (new / rz) * p
            rz = new
        return x

    def mme(self, y, tol=TOL):
        S = self.solve(torch.cat([self.X, y], 1), tol)
        inv = torch.linalg.inv(self.X.T @ S[:, :-1])
        beta = inv @ (self.X.T @ S[:, -1:])
        vr = S[:, -1:] - S[:, :-1] @ beta
        return S[:, :-1], inv, beta, vr, self.vc[1] * self.A.apply(self.sums(vr))


def exact(case, seed):
    kind, N = case["kind"], case["N"]
    if kind == "aireml":        # a whole run: dozens of solves, its probes drawn on the GPU
        return None
    if kind == "dense":
        A = _DenseA(_grm(case, seed), N)
    else:
        bed = _bed(case, seed)
        A = _Zs(bed, N)
    if kind == "apply":
        return (VC[1] * A.apply(torch.from_numpy(np.ascontiguousarray(_z(case, seed))).to(DEV))).cpu().numpy()
    if kind == "load":
        return [A.diag(), A.M]
    if kind == "build":
        out = torch.zeros((N, N), dtype=torch.float64, device=DEV)
        for z in A.chunks():
            out.addmm_(z.T, z)
        out /= max(1, A.M)
        return out[torch.ones((N, N), dtype=torch.bool, device=DEV).tril_()]
    if kind in ("pcg", "eval") and N * case["M"] > 1.2e10:
        return None             # minutes in float64
    indiv, X, y = _cohort(case, seed, _signal(case, bed, seed) if kind != "dense" else None)
    m = _Model(A, indiv, X, N, THETA0 if kind == "eval" else VC)
    if kind in ("pcg", "dense"):
        return m.solve(_rhs(case, X, y, seed).T.contiguous()).T.contiguous()
    y = torch.from_numpy(y).to(DEV)[:, None]
    if kind == "mme":
        _, _, beta, vr, uhat = m.mme(y)
        s0, s1 = m.sums(vr), m.sums(m.t * vr)
        bhat = torch.cat([VC[2] * s0 + VC[3] * s1, VC[3] * s0 + VC[4] * s1], 1).reshape(-1)
        return [beta[:, 0], uhat[:, 0], bhat, vr[:, 0]]
    # eval: the terms that take no probes
    VX, inv, _, vr, uhat = m.mme(y)
    w, tw = m.sums(vr)[m.i], m.sums(m.t * vr)[m.i]
    F = torch.cat([vr, uhat[m.i] / THETA0[1], w, m.t * w + tw, m.t * tw], 1)
    S = m.solve(F)
    ai = 0.5 * F.T @ (S - VX @ (inv @ (m.X.T @ S)))
    return [(vr.T @ F)[0], None, None, ai]
