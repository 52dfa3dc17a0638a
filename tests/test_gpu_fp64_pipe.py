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
