"""The record kernels of a solve (k_solve.cu) at the edges of their layouts: individuals of 1 to 700
records (one thread up to 256, a CTA above), 1 to 130 columns (tiles of at most 128), masking, both
arithmetics, the three start points."""
import numpy as np
import pytest

import globe_gb300 as G
from helpers import VC_F, cohort, rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(orc):
    counts = np.array([1, 2, 3, 255, 700, 1, 256, 257, 4, 5, 9, 300, 6, 48, 49, 1, 8] + [2, 7, 1, 4] * 9)
    N = len(counts)
    rng = np.random.default_rng(3)
    indiv = np.repeat(np.arange(N, dtype=np.int32), counts)
    X = np.column_stack([np.ones(len(indiv)), rng.standard_normal(len(indiv)), rng.uniform(0, 2, len(indiv))])
    y = rng.standard_normal(len(indiv))
    packed = cohort(4, N, 300, recs=("uniform", 1, 2), miss=0.02)["packed"]
    with G.Context(0) as ctx:
        ctx.load_records(indiv, X, y, N)
        ctx.load_bed(packed)
        ctx.set_vc(VC_F)
        s = orc.Solver(indiv, X, y, N, VC_F, packed=packed)
        s.precond_build()
        yield ctx, s, rng.standard_normal((len(indiv), 130)) * np.logspace(-3, 3, 130)


# both sides stop at a relative residual of 1e-11; V's condition number here is below 1e2
@pytest.mark.parametrize("prec", [G.PREC_FP64, G.PREC_MIXED])
@pytest.mark.parametrize("k", [1, 5, 33, 65, 128, 129, 130])
def test_columns_and_block_lengths(setup, k, prec):
    ctx, s, B = setup
    ref, _ = s.pcg(B[:, :k], 1e-11, rule=1)
    for mask in (False, True):
        X, info = ctx.pcg(B[:, :k], tol=1e-11, rule=G.RULE_AIREML, mask=mask, precision=prec)
        assert info["converged"]
        assert max(rel(X[:, c], ref[:, c]) for c in range(k)) < 1e-9


@pytest.mark.parametrize("prec", [G.PREC_FP64, G.PREC_MIXED])
def test_start_points_zero_columns_and_no_iterations(setup, prec):
    ctx, s, B = setup
    B = B[:, :7].copy()
    B[:, 3] = 0.0
    ref, _ = s.pcg(B[:, [0, 1, 2, 4, 5, 6]], 1e-11, rule=1)
    x0 = np.random.default_rng(5).standard_normal(B.shape)
    for kw in (dict(), dict(x0mode=G.X0_PRECOND), dict(X0=x0)):
        X, info = ctx.pcg(B, tol=1e-11, rule=G.RULE_AIREML, precision=prec, **kw)
        assert info["converged"] and not X[:, 3].any()
        assert rel(X[:, [0, 1, 2, 4, 5, 6]], ref) < 1e-9
    X, info = ctx.pcg(B, X0=x0, maxit=0, precision=prec)       # no iteration: the start point comes back
    keep = [0, 1, 2, 4, 5, 6]
    assert info["iters"] == 0 and rel(X[:, keep], x0[:, keep]) < 1e-13 and not X[:, 3].any()
