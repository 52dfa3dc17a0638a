"""A_ii from the genotypes (k_geno_diag) against a sum in extended precision, at the edges of its 8-SNP steps, 128-SNP
blocks, 128-individual chunks and 16384-individual CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# zs^2 carries a few units of 2^-53 (division, square root, square), all terms are non-negative, and
# the fixed-point sum is within M 2^-63 of the largest possible one
TOL = 1e-14


@pytest.mark.parametrize("N,M", [(2, 1), (5, 7), (16, 8), (127, 9), (128, 127), (129, 128), (130, 1025), (16383, 65),
                                 (16384, 130), (16385, 143), (33001, 72), (40, 20011)])
def test_matches_exact_sum(gctx, N, M):
    rng = np.random.default_rng(N + M)
    packed = rng.integers(0, 256, (M, (N + 3) // 4), dtype=np.uint8)
    gctx.load_records(np.arange(N, dtype=np.int32), np.zeros((N, 1)) + 1.0, rng.standard_normal(N), N)
    gctx.load_bed(packed, min_maf=0.0, max_miss=1.0)
    codes = ((packed[:, :, None] >> (2 * np.arange(4, dtype=np.uint8))) & 3).reshape(M, -1)[:, :N]
    g = np.array([2.0, 0.0, 1.0, 0.0])[codes]
    obs = (codes != 1).sum(1).astype(np.float64)
    f = np.where(obs > 0, g.sum(1) / np.maximum(2.0 * obs, 1.0), 0.0)
    den = 2.0 * f * (1.0 - f)
    inv = np.where(den > 1e-12, 1.0 / np.sqrt(np.maximum(den, 1e-300)), 1.0)
    zs = (np.array([2.0, 0.0, 1.0, 0.0])[None, :] - 2.0 * f[:, None]) * inv[:, None]
    want = np.take_along_axis((zs * zs).astype(np.longdouble), codes.astype(np.int64), 1).sum(0) / M
    assert np.abs(gctx.genetic_diag() - want).max() <= TOL * want.max()


def test_reload_takes_over_the_genotype_copy(gctx):
    """A second load of about the same size, of a smaller one and of a larger one give what a first
    load gives, whether the memory of the earlier copy is taken over or not."""
    import globe_gb300 as G
    rng = np.random.default_rng(5)
    N = 1000
    packed = rng.integers(0, 256, (9000, N // 4), dtype=np.uint8)
    z = rng.standard_normal((N, 6))
    with G.Context(0) as fresh:
        for M in (8000, 7700, 7100, 900, 9000):
            out = []
            for ctx in (gctx, fresh):
                if M == 8000 or ctx is fresh:
                    ctx.load_records(np.arange(N, dtype=np.int32), np.ones((N, 1)), z[:, 0], N)   # drops the copy
                ctx.load_bed(packed[:M], min_maf=0.0, max_miss=1.0)
                ctx.set_vc((0.6, 0.4, 0.4, 0.2, 0.2))
                ctx.set_precision(G.PREC_MIXED)
                out.append((ctx.genetic_diag(), ctx.grm_apply(z)))
                ctx.set_precision(G.PREC_FP64)
            assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1]), M
