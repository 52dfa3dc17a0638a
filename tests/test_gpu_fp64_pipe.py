"""The small FP64 products (k_geno_p1, k_geno_p2, k_sum_splits) against the oracle: every number of warps
per two SNPs, odd SNP counts, one to eight columns and past them."""
import numpy as np
import pytest

import globe_gb300 as G
from helpers import VC_F, cohort, rel

pytestmark = pytest.mark.gpu

# sqrt(N) + sqrt(M) units of 2^-53 of a column at most (~4e-14)
TOL = 1e-13


@pytest.mark.parametrize("N,M", [(3, 40), (31, 1), (129, 601), (257, 601), (601, 1503), (2000, 129), (1025, 5001)])
def test_small_products(gctx, orc, N, M):
    c = cohort(90 + N, N, M, recs=("uniform", 1, 2), miss=0.03)
    indiv = c["indiv"].astype(np.int32)
    gctx.load_records(indiv, c["X"], c["y"], N)
    gctx.load_bed(c["packed"])
    gctx.set_vc(VC_F)
    gctx.set_precision(G.PREC_FP64)
    s = orc.Solver(indiv, c["X"], c["y"], N, VC_F, packed=c["packed"])
    rng = np.random.default_rng(N)
    for k in (1, 2, 4, 7, 9):
        Z = rng.standard_normal((N, k))
        got, ref = gctx.grm_apply(Z), s.grm_apply(Z)
        assert max(rel(got[:, q], ref[:, q]) for q in range(k)) < TOL, k


# either side of the sizes at which an FP64 solve's products change path (5e6 in N M k for one or
# two columns, 5e5 for more); residuals of 1e-12 leave solutions of these cohorts within 1e-9
@pytest.mark.parametrize("N,M,k", [(1000, 4900, 1), (1000, 5300, 1), (1000, 2450, 2), (1000, 2700, 2), (300, 540, 3),
                                   (300, 600, 3)])
def test_solves_either_side_of_the_threshold(gctx, orc, N, M, k):
    c = cohort(70 + k, N, M, recs=("uniform", 1, 4), miss=0.02)
    indiv = c["indiv"].astype(np.int32)
    gctx.load_records(indiv, c["X"], c["y"], N)
    gctx.load_bed(c["packed"])
    gctx.set_vc(VC_F)
    s = orc.Solver(indiv, c["X"], c["y"], N, VC_F, packed=c["packed"])
    s.precond_build()
    B = np.asfortranarray(np.random.default_rng(k).standard_normal((len(indiv), k)))
    X, info = gctx.pcg(B, tol=1e-12, rule=G.RULE_PCGSOLVER)
    Xo, it = s.pcg(B, 1e-12, rule=0)
    assert rel(X, Xo) < 1e-9 and info["iters"] == it
