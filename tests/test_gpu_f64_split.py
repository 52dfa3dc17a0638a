"""GLOBE_PREC_FP64 products on the tensor cores (12 base-32 digits, exact sums) against the FP64
oracle and against the FP64-pipe kernels, which run the smaller products.

A single operator call takes the tensor cores from N Mk k = 4e7 on (geno_apply_f64), N N k = 4e6
with a dense GRM (dense_apply_f64)."""
import numpy as np
import pytest

import globe_gb300 as G
from helpers import VC_F, cohort, rel

pytestmark = pytest.mark.gpu

# the oracle's FP64 sums are within sqrt(N) + sqrt(M) units of 2^-53 of a column (~2e-14 at these
# sizes); the digit product within a few units
TOL = 1e-13


def _load(gctx, orc, N, M, seed):
    c = cohort(seed, N, M, recs=("uniform", 1, 2), miss=0.03, edge=True)
    indiv = c["indiv"].astype(np.int32)
    gctx.load_records(indiv, c["X"], c["y"], N)
    gctx.load_bed(c["packed"])
    gctx.set_vc(VC_F)
    gctx.set_precision(G.PREC_FP64)
    return orc.Solver(indiv, c["X"], c["y"], N, VC_F, packed=c["packed"])


# tiles of 512, 256 and 128 rows, K stages of 128, one row or column past them, one to three groups
@pytest.mark.parametrize("N,M,ks", [(2049, 4001, (5, 16, 17, 22, 45)), (513, 16500, (5, 6)), (16385, 531, (5, 10)),
                                    (6500, 6600, (1, 2))])
def test_matches_oracle_and_fp64_pipe(gctx, orc, N, M, ks):
    s = _load(gctx, orc, N, M, 50 + N)
    rng = np.random.default_rng(M)
    for k in ks:
        Z = rng.standard_normal((N, k)) * np.logspace(-8, 8, k)
        Z[:, 0] += 30.0                                   # a mean that the centring cancels
        if k > 4:
            Z[:, 2] = np.exp(2 * rng.standard_normal(N))
            Z[:, 3] = np.eye(N)[N // 2]
            Z[:, 4] = 0.0
        got, ref = gctx.grm_apply(Z), s.grm_apply(Z)
        assert max(rel(got[:, c], ref[:, c]) for c in range(k) if ref[:, c].any()) < TOL, k
        if k > 4:
            assert not got[:, 4].any()
        if N * M < 3e7:                                   # one column alone runs on the FP64 pipe
            assert rel(got[:, 1], gctx.grm_apply(Z[:, 1])[:, 0]) < TOL, k


def test_column_magnitudes_and_nonfinite(gctx, orc):
    """Columns near either end of the range of a double are scaled exactly; a column holding a NaN
    or an infinity gives NaN and leaves the others alone."""
    N, M = 2049, 4001
    s = _load(gctx, orc, N, M, 7)
    z = np.random.default_rng(1).standard_normal(N)
    Z = np.column_stack([z, z * 2.0 ** 960, z * 2.0 ** -960, z, z, z])
    Z[3, 3], Z[5, 4] = np.nan, -np.inf
    got = gctx.grm_apply(Z)
    assert rel(got[:, 0], s.grm_apply(z[:, None])[:, 0]) < TOL
    assert np.array_equal(got[:, 1], got[:, 0] * 2.0 ** 960) and np.array_equal(got[:, 2], got[:, 0] * 2.0 ** -960)
    assert np.isnan(got[:, 3:5]).all() and np.array_equal(got[:, 5], got[:, 0])
    sub = gctx.grm_apply(np.column_stack([z * 2.0 ** -1040] * 6))
    assert np.allclose(sub[:, 2], got[:, 0] * 2.0 ** -1040, rtol=0, atol=N * 2.0 ** -1074)


def test_solve_repeats_and_masks(gctx, orc):
    """FP64 solves on the digit products: graphs, the device loop and direct launches give the same
    bits, with and without masking, and the oracle's solution."""
    s = _load(gctx, orc, 901, 2300, 11)
    B = np.random.default_rng(2).standard_normal((s.Nrec, 6)) * [1, 1e3, 1e-3, 1, 5, 1]
    s.precond_build()
    ref, _ = s.pcg(B, 1e-11, rule=1)
    for mask in (False, True):
        out = []
        try:
            for graphs, loop in ((False, False), (True, False), (True, True)):
                gctx.set_graphs(graphs)
                gctx.set_device_loop(loop)
                out.append(gctx.pcg(B, tol=1e-11, rule=G.RULE_AIREML, mask=mask)[0])
        finally:
            gctx.set_graphs(True)
            gctx.set_device_loop(True)
        assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
        assert max(rel(out[0][:, c], ref[:, c]) for c in range(6)) < 1e-9


def _dense(gctx, N, seed, shrink=None):
    rng = np.random.default_rng(seed)
    W = rng.standard_normal((800, N))
    A = (W.T @ W / 800).astype(np.float32)
    if shrink is not None:                                # one individual on a much smaller scale
        A[shrink] *= np.float32(1e-6)
        A[:, shrink] *= np.float32(1e-6)
    lt = A[np.tril_indices(N)]
    gctx.load_records(np.arange(N, dtype=np.int32), np.ones((N, 1)), np.zeros(N), N)
    gctx.load_grm(lt, N)
    gctx.set_vc(VC_F)
    gctx.set_precision(G.PREC_FP64)
    low = np.tril(A.astype(np.float64))
    return low + np.tril(low, -1).T


# row tiles of 256 and K chunks of 128, one past them; one to three column groups
@pytest.mark.parametrize("N,ks", [(2049, (1, 5)), (901, (5, 16)), (640, (10, 21, 22, 43)), (385, (28,))])
def test_dense_matches_float64(gctx, N, ks):
    A = _dense(gctx, N, N)
    rng = np.random.default_rng(1)
    for k in ks:
        Z = rng.standard_normal((N, k)) * np.logspace(-200, 200, k)
        if k > 4:
            Z[:, 2] = np.exp(2 * rng.standard_normal(N))
            Z[:, 3] = 0.0
        got, ref = gctx.grm_apply(Z), VC_F[1] * (A @ Z)
        # FP64 sums of N terms: sqrt(N) units of 2^-53
        assert max(rel(got[:, c] / np.abs(Z[:, c]).max(), ref[:, c] / np.abs(Z[:, c]).max())
                   for c in range(k) if ref[:, c].any()) < 1e-14, k
        assert k <= 4 or not got[:, 3].any()


def test_dense_small_row_keeps_its_digits(gctx):
    """A row far below max|A| would lose digits on the planes' common grid: the FP64 pipe runs."""
    N, i = 2049, 77
    A = _dense(gctx, N, 3, shrink=i)
    Z = np.random.default_rng(2).standard_normal((N, 2))
    Z[i] = 0.0
    got, ref = gctx.grm_apply(Z), VC_F[1] * (A @ Z)
    assert np.abs(got[i] / ref[i] - 1).max() < 1e-11 and rel(got, ref) < 1e-13


def test_dense_precisions_hold_their_own_planes(gctx):
    """Mixed products between FP64 ones: each precision gives the same bits throughout."""
    _dense(gctx, 901, 4)
    Z = np.random.default_rng(3).standard_normal((901, 6))
    out = {}
    try:
        for prec in (G.PREC_MIXED, G.PREC_FP64, G.PREC_MIXED, G.PREC_FP64):
            gctx.set_precision(prec)
            out.setdefault(prec, []).append(gctx.grm_apply(Z))
    finally:
        gctx.set_precision(G.PREC_FP64)
    assert all(np.array_equal(a, b) for a, b in out.values())
    assert 0 < rel(out[G.PREC_MIXED][0], out[G.PREC_FP64][0]) < 1e-9
