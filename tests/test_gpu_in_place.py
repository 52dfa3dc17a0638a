"""GRM products whose output takes the place of their input (d_out == d_Z of globe_grm_apply_dev)."""
import ctypes as C

import numpy as np
import pytest

import globe_gb300 as G
from helpers import VC_F, cohort

pytestmark = pytest.mark.gpu


# N Mk k = 4e7 and more takes the tensor cores in FP64; 9 columns and more are the ones whose grouping
# is timed on the first product of a shape, one shape a case
@pytest.mark.parametrize("prec,k", [(G.PREC_FP64, 10), (G.PREC_FP64, 23), (G.PREC_FP64, 4), (G.PREC_MIXED, 11)])
def test_first_product_of_a_shape_in_place(gctx, prec, k):
    import torch
    N, M = 1100 + k, 5003
    c = cohort(60 + k, N, M, recs=("uniform", 1, 2), miss=0.02)
    gctx.load_records(c["indiv"].astype(np.int32), c["X"], c["y"], N)
    gctx.load_bed(c["packed"])
    gctx.set_vc(VC_F)
    gctx.set_precision(prec)
    try:
        z = torch.from_numpy(np.random.default_rng(k).standard_normal((k, N))).cuda()
        buf, out = z.clone(), torch.empty_like(z)
        torch.cuda.synchronize()
        for src, dst in ((buf, buf), (z, out), (z, out)):     # in place first: the shape is not tuned yet
            assert gctx._L.globe_grm_apply_dev(gctx.h, C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()), k) == 0
        torch.cuda.synchronize()
        assert torch.equal(buf, out)
    finally:
        gctx.set_precision(G.PREC_FP64)
