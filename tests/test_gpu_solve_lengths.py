"""Who walks an individual's records in a solve (shape() in k_solve.cu): one thread, a team of a CTA's
threads or a whole CTA, at the record counts where that changes, in cohorts of one kind and of all."""
import numpy as np
import pytest

import globe_gb300 as G
from helpers import VC_F, cohort, rel

pytestmark = pytest.mark.gpu

EDGES = [31, 32, 33, 34, 63, 64, 65, 127, 128, 129, 255, 256, 257, 258, 1, 5, 513]
# name -> (record counts, columns): one thread takes 32 to 89 records here, by the size of the solve
COHORTS = {
    "edges": (EDGES + [3, 7] * 5, (1, 5, 129)),
    "all-long": ([33 + (7 * i) % 40 for i in range(700)], (1, 5, 129)),   # teams only, several steps of a CTA
    "all-very-long": ([260 + i for i in range(40)], (1, 5, 129)),           # whole CTAs only
    "none-long": ([1 + (5 * i) % 32 for i in range(900)], (1, 5, 129)),
    # 390 columns leave teams of two, of which each may take half of an odd limit
    "two-a-team": ([65, 66, 67, 68] * 20 + [69, 70, 71, 30, 31] * 11, (390,)),
    "mixed": ([300, 290] + [60 + (11 * i) % 50 for i in range(900)] + [2, 9] * 300, (1, 20, 33)),
}


def _load(ctx, orc, counts):
    N = len(counts)
    rng = np.random.default_rng(N)
    counts = rng.permutation(counts)
    indiv = np.repeat(np.arange(N, dtype=np.int32), counts)
    X = np.column_stack([np.ones(len(indiv)), rng.uniform(0, 2, len(indiv))])
    y = rng.standard_normal(len(indiv))
    packed = cohort(4, N, 300, recs=("uniform", 1, 2), miss=0.02)["packed"]
    ctx.load_records(indiv, X, y, N)
    ctx.load_bed(packed)
    ctx.set_vc(VC_F)
    s = orc.Solver(indiv, X, y, N, VC_F, packed=packed)
    s.precond_build()
    return s, rng.standard_normal((len(indiv), 390))


# both sides stop at a relative residual of 1e-11; with up to 513 records an individual V's condition
# number stays below 1e3
@pytest.mark.parametrize("name", sorted(COHORTS))
def test_lengths_match_oracle(gctx, orc, name):
    counts, ks = COHORTS[name]
    s, B = _load(gctx, orc, counts)
    ref, _ = s.pcg(B[:, :max(ks)], 1e-11, rule=1)
    for k in ks:
        for prec in (G.PREC_FP64, G.PREC_MIXED):
            X, info = gctx.pcg(B[:, :k], tol=1e-11, rule=G.RULE_AIREML, precision=prec)
            assert info["converged"]
            assert max(rel(X[:, c], ref[:, c]) for c in range(k)) < 1e-8, (name, k, prec)


# 1216 pairs of threads at 128 columns: 16 individuals each, so their sums pass from double-float into FP64
# twice.  Residuals of a few per cent, r recurred in 47 bits from |V p| < 1e3 |p|
@pytest.mark.parametrize("k", [1, 128])
def test_sums_over_many_individuals_a_thread(gctx, k):
    N = 20011
    rng = np.random.default_rng(N)
    counts = rng.integers(1, 4, N)
    indiv = np.repeat(np.arange(N, dtype=np.int32), counts)
    X = np.column_stack([np.ones(len(indiv)), rng.uniform(0, 2, len(indiv))])
    gctx.load_records(indiv, X, rng.standard_normal(len(indiv)), N)
    gctx.load_bed(rng.integers(0, 256, (130, (N + 3) // 4), dtype=np.uint8), min_maf=0.0, max_miss=1.0)
    gctx.set_vc(VC_F)
    B = rng.standard_normal((len(indiv), k))
    for prec in (G.PREC_FP64, G.PREC_MIXED):
        Y, info = gctx.pcg(B, tol=0.0, maxit=4, rule=G.RULE_AIREML, precision=prec)
        r = np.linalg.norm(B - gctx.vx(Y), axis=0) / np.linalg.norm(B, axis=0)
        assert info["iters"] == 4 and 1e-6 < r.max() < 1
        assert abs(info["max_rel_res"] / r.max() - 1) < 1e-8
