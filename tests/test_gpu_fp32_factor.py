"""FP32 products whose constant output factor lies outside 2^-120 .. 2^120
while their results do not: unscaled products, and the scaled ones inside a
mixed solve, of the full x-ANNNI and DNNI operators at large betaJ.

Bars: FP32 2e-5 of max|y| (as the other products), mixed eigenvalues 1e-10 of
the FP64 mode's.
"""
import numpy as np
import pytest

import latttmat_gb300 as lt
from cases import seeded_input
from gpu_util import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
oracle = pytest.importorskip("oracle.oracle")


# output factors e^{-KL(1-kappa)} = e^-96, e^-86 (x-ANNNI); nf = e^{-2KL(1-kappa)} = e^-112, e^-105 (DNNI)
@pytest.mark.parametrize("args", [("A", 2, 1, 6.0, 0.0, 0.0, 16, 0.0, 0), ("A", 2, 1, 9.0, 0.2, 0.05, 12, 0.0, 0),
                                  ("D", 2, 2, 4.0, 0.0, 0.0, 14, 0.0, 0), ("D", 2, 2, 5.0, 0.125, 0.05, 12, 0.0, 0)])
def test_unscaled_products(args):
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    x = seeded_input(op.rows(), 4).astype(np.float32)
    xd = torch.tensor(x, device="cuda")
    yd = torch.empty_like(xd)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    op.perform_op_dev(xd.data_ptr(), yd.data_ptr(), lt.TM_F32, s.cuda_stream)
    torch.cuda.synchronize()
    assert rel_err(yd.double().cpu().numpy(), ref.perform_op(x.astype(np.float64))) < 2e-5


# what is left of the output factor in a scaled product, e^{-KL(2-kappa)} (x-ANNNI) or e^{-2KL(1-kappa)}
# (DNNI): e^-88, e^-85, e^-88, e^-90
@pytest.mark.parametrize("args", [("A", 2, 1, 2.2, 0.0, 0.05, 20, 0.0, 0), ("A", 2, 1, 2.5, 0.3, 0.05, 20, 0.0, 0),
                                  ("D", 2, 2, 2.2, 0.0, 0.05, 20, 0.0, 0), ("D", 2, 2, 2.5, 0.0, 0.05, 18, 0.0, 0)])
def test_mixed_solves(args):
    op = lt.TMatOp(*args)
    v64, _, _, i64 = op.eigs(1, tol=1e-10, mode=lt.TM_EIGS_F64)
    vm, _, _, im = op.eigs(1, tol=1e-10, mode=lt.TM_EIGS_MIXED)
    assert i64["nconv"] == 1 and im["nconv"] == 1
    np.testing.assert_allclose(vm, v64, rtol=1e-10)
