"""Memory that only makes later calls faster (the second genotype copy and the digit planes of FP64
products, the tensor-core workspaces) is given back where an allocation of the context needs it."""
import contextlib

import numpy as np
import pytest

import globe_gb300 as G
from helpers import VC_F, rel

pytestmark = pytest.mark.gpu

LEAVE = 96 << 20


@contextlib.contextmanager
def _filled():
    """All but ~LEAVE bytes of the device, as another library of the process would hold it."""
    import torch
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(max(0, free - LEAVE), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del fill
        torch.cuda.empty_cache()


def _context(ctx, kind):
    rng = np.random.default_rng(3)
    N, M = (6007, 100) if kind == "dense" else (10007, 60000)
    t = rng.uniform(0, 2, N)
    ctx.load_records(np.arange(N, dtype=np.int32), np.column_stack([np.ones(N), t]), rng.standard_normal(N), N)
    if kind == "dense":
        W = rng.standard_normal((M, N)).astype(np.float32)
        A = W.T @ W / np.float32(M)
        ctx.load_grm(A[np.tril_indices(N)], N)
    else:
        ctx.load_bed(rng.integers(0, 256, (M, (N + 3) // 4), dtype=np.uint8), min_maf=0.0, max_miss=1.0)
    ctx.set_vc(VC_F)
    return N, rng


@pytest.mark.parametrize("kind", ["dense", "genotypes"])
def test_fp64_copies_make_room(kind):
    """V x of more columns than fit beside the copies that the first, small product made."""
    with G.Context(0) as ctx:
        N, rng = _context(ctx, kind)
        x = rng.standard_normal((N, 8))
        ref = ctx.vx(x)                                   # on the tensor cores: planes or copy made
        held = ctx.device_bytes()
        wide = np.asfortranarray(np.tile(x, (1, 400 // 8 if kind == "dense" else 30)))
        with _filled():
            got = ctx.vx(wide)                            # five N x k workspaces and a quarter each
        assert rel(got, np.tile(ref, (1, got.shape[1] // 8))) < 1e-12
        assert ctx.device_bytes() < held + 5 * 1.3 * wide.nbytes
        assert rel(ctx.vx(x), ref) < 1e-12


def test_build_workspaces_make_room():
    """The GRM build's workspaces give way to a solve's vectors; the next build gets them again."""
    with G.Context(0) as ctx:
        N, rng = _context(ctx, "genotypes")
        ctx.set_precision(G.PREC_MIXED)
        lt = ctx.grm_build()
        ctx.set_precision(G.PREC_FP64)
        with _filled():
            X = ctx.vx(rng.standard_normal((N, 240)))
        assert np.isfinite(X).all()
        ctx.set_precision(G.PREC_MIXED)
        assert np.array_equal(ctx.grm_build(), lt)
