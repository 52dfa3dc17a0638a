"""A_ii of each individual where a few rare SNPs have squares of standardised genotypes far above the
rest's: the fixed-point sum's step (k_geno_diag) follows the sum of the SNPs' largest squares."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M,rare", [(2000, 20000, 5), (2000, 20000, 1), (601, 9000, 0), (3001, 3000, 3000)])
def test_each_individual(gctx, N, M, rare):
    rng = np.random.default_rng(N + rare)
    codes = rng.choice([0, 2, 3, 1], (M, N), p=[0.2, 0.4, 0.38, 0.02]).astype(np.uint8)   # 2, 1, 0 copies, missing
    for s in rng.choice(M, rare, replace=False):
        codes[s] = 3
        codes[s, rng.integers(N)] = 2                     # one carrier
    full = np.zeros((M, (N + 3) // 4 * 4), np.uint8)
    full[:, :N] = codes
    packed = full[:, 0::4] | full[:, 1::4] << 2 | full[:, 2::4] << 4 | full[:, 3::4] << 6
    gctx.load_records(np.arange(N, dtype=np.int32), np.ones((N, 1)), rng.standard_normal(N), N)
    gctx.load_bed(packed, min_maf=0.0, max_miss=1.0)
    copies = np.array([2.0, 0.0, 1.0, 0.0])
    obs = (codes != 1).sum(1).astype(np.float64)
    f = copies[codes].sum(1) / (2.0 * obs)
    den = 2.0 * f * (1.0 - f)
    zs = (copies[None, :] - 2.0 * f[:, None]) / np.sqrt(den)[:, None]
    sq = (zs * zs).astype(np.longdouble)
    want = np.zeros(N, np.longdouble)
    for s0 in range(0, M, 1000):
        want += np.take_along_axis(sq[s0:s0 + 1000], codes[s0:s0 + 1000].astype(np.int64), 1).sum(0)
    want /= M
    # half a step, its step 2^-61 of the bound at most; a few units of 2^-53 in each square, on both sides
    step = 2.0 ** -61 * np.ceil((zs * zs)[:, :3].max(1)).sum()
    got = gctx.genetic_diag()
    assert (np.abs(got - want) <= 0.5 * step + 16 * 2.0 ** -53 * want).all()
