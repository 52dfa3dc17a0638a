"""FP64 products of a dense GRM row by row: matrices with zeros between families and right-hand sides
whose magnitude differs between them, where a column's largest entry says nothing about a row."""
import ctypes as C

import numpy as np
import pytest

import globe_gb300 as G
from helpers import VC_F

pytestmark = pytest.mark.gpu

FAM = 40        # individuals a family
# FP64 sums of at most FAM terms of magnitude |a z|, each product and sum within 2^-53, and the final scaling
TOL = (FAM + 3) * 2.0 ** -53


def _families(ctx, N, seed, small=None):
    """Block-diagonal A with families of FAM; small: a magnitude of entries put between families."""
    rng = np.random.default_rng(seed)
    A = np.zeros((N, N), np.float32)
    for s in range(0, N, FAM):
        W = rng.standard_normal((60, min(FAM, N - s)))
        A[s:s + FAM, s:s + FAM] = W.T @ W / 60
    if small:
        for i in range(0, N - FAM, 7):
            A[i, i + FAM] = A[i + FAM, i] = small * (1 + i / N)
    ctx.load_records(np.arange(N, dtype=np.int32), np.ones((N, 1)), np.zeros(N), N)
    low = np.tril(A.astype(np.float64))
    ctx.load_grm(A[np.tril_indices(N)], N)
    ctx.set_vc(VC_F)
    ctx.set_precision(G.PREC_FP64)
    return low + np.tril(low, -1).T


def _want(A, Z):
    return VC_F[1] * (A.astype(np.longdouble) @ Z.astype(np.longdouble)), VC_F[1] * (np.abs(A) @ np.abs(Z))


# range of the families' magnitudes: inside 16 digits' 80 bits, at their edge, past them
@pytest.mark.parametrize("decades", [0, 6, 8, 12, 30])
@pytest.mark.parametrize("N,k", [(2049, 1), (901, 5), (641, 16), (700, 37)])
def test_rows_of_families_of_any_magnitude(gctx, N, k, decades):
    A = _families(gctx, N, N)
    rng = np.random.default_rng(k)
    Z = rng.standard_normal((N, k)) * 10.0 ** -rng.uniform(0, decades, N)[:, None] if decades else rng.standard_normal((N, k))
    Z[::13, 0] = 0.0
    got = gctx.grm_apply(Z)
    want, size = _want(A, Z)
    assert (np.abs(got - want) <= TOL * size).all()


# what the digits leave of a few entries is added: 1 to 8 in one range of rows, in several, past 8 (then the
# whole column is formed anew), and of the smallest magnitudes
@pytest.mark.parametrize("rows", [[3], [40, 41, 42, 43, 44, 45, 46, 47], [80, 81, 82, 83, 84, 85, 86, 87, 88],
                                  [0, 1023, 1024, 2048], list(range(5, 2049, 130))])
@pytest.mark.parametrize("small", [1e-9, 1e-40])
def test_rows_of_a_few_small_entries(gctx, rows, small):
    N = 2049
    A = _families(gctx, N, 10)
    rng = np.random.default_rng(len(rows))
    Z = rng.standard_normal((N, 9))
    Z += np.sign(Z) * 0.5                              # the others are within 2^4 of the largest
    for r in rows:                                     # a family of its own scale each
        Z[r // FAM * FAM:r // FAM * FAM + FAM, 1::2] = 0.0
    for r in rows:
        Z[r, 1::2] = small * rng.standard_normal(4)
    got = gctx.grm_apply(Z)
    want, size = _want(A, Z)
    assert (np.abs(got - want) <= TOL * size).all()
    assert np.array_equal(got, gctx.grm_apply(Z))


# the smaller families' entries pass below the smallest double when the column is scaled
@pytest.mark.parametrize("big,small", [(1e300, 1e-60), (1e300, 1e-120), (1e280, 1e-300)])
def test_rows_across_the_range_of_a_double(gctx, big, small):
    N = 2049
    A = _families(gctx, N, 9)
    Z = np.random.default_rng(6).standard_normal((N, 2))
    Z[:, 0] *= np.where(np.arange(N) // FAM % 2, big, small)
    got = gctx.grm_apply(Z)
    want, size = _want(A, Z)
    assert (np.abs(got - want) <= TOL * size + 2.0 ** -1074).all()


# entries that the least number of planes does not hold exactly; that no number of them does
@pytest.mark.parametrize("small", [1e-9, 3e-12, 1e-13, 1e-16, 1e-30])
def test_rows_with_small_entries_of_a(gctx, small):
    N = 2049
    A = _families(gctx, N, 3, small)
    Z = np.random.default_rng(1).standard_normal((N, 2))
    Z[::FAM] *= 1e6
    got = gctx.grm_apply(Z)
    want, size = _want(A, Z)
    assert (np.abs(got - want) <= TOL * size).all()


def test_nonfinite_entries_reach_the_rows_that_they_enter(gctx):
    """A z as FP64 sums give it: an infinity of a family is one in its rows, and 0 times it NaN elsewhere."""
    N = 901
    A = _families(gctx, N, 5)
    Z = np.random.default_rng(2).standard_normal((N, 6))
    ref = gctx.grm_apply(Z)
    Z[50, 1], Z[7, 3], Z[8, 4] = np.inf, -np.inf, np.nan
    got = gctx.grm_apply(Z)
    assert np.array_equal(got[:, [0, 2, 5]], ref[:, [0, 2, 5]]) and np.isnan(got[:, 4]).all()
    for c, r, v in ((1, 50, np.inf), (3, 7, -np.inf)):
        rows = A[r] != 0
        assert np.array_equal(got[rows, c], v * np.sign(A[r, rows])) and np.isnan(got[~rows, c]).all()


def test_in_place_and_repeated(gctx):
    import torch
    N, k = 901, 11
    _families(gctx, N, 6)
    rng = np.random.default_rng(4)
    Z = rng.standard_normal((k, N)) * 10.0 ** -rng.uniform(0, 20, N)
    z = torch.from_numpy(Z).cuda()
    buf, out = z.clone(), torch.empty_like(z)
    torch.cuda.synchronize()
    for src, dst in ((z, out), (buf, buf)):
        assert gctx._L.globe_grm_apply_dev(gctx.h, C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()), k) == 0
    torch.cuda.synchronize()
    assert torch.equal(buf, out)


def test_solve_with_wide_columns_repeats(gctx):
    """Direct launches, graphs and the device loop give the same bits where columns go to the FP64 pipe."""
    N = 901
    A = _families(gctx, N, 8)
    rng = np.random.default_rng(5)
    B = rng.standard_normal((N, 6)) * 10.0 ** -rng.uniform(0, 14, N)[:, None]
    out = []
    try:
        for graphs, loop in ((False, False), (True, False), (True, True)):
            gctx.set_graphs(graphs)
            gctx.set_device_loop(loop)
            out.append(gctx.pcg(B, tol=1e-12, rule=G.RULE_AIREML)[0])
    finally:
        gctx.set_graphs(True)
        gctx.set_device_loop(True)
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    X = out[0]                                       # one record an individual at time 1: V = sig2g A + c I
    c = VC_F[0] + VC_F[2] + 2 * VC_F[3] + VC_F[4]
    r = B - (VC_F[1] * A @ X + c * X)
    assert (np.linalg.norm(r, axis=0) <= 1e-11 * np.linalg.norm(B, axis=0)).all()
