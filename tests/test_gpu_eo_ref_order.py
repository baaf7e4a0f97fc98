"""Even/odd products on vectors in the reference's order: the permutation is
folded into the input scaling, FP32 outputs are scaled in double-float where
the scales fit the FP32 exponent range and in FP64 elsewhere.

Bars: FP64 / double-float 1e-12 of max|y|; FP32 2e-5 of max|y|, as the other
products.  Scaling x by a power of two scales every FP32 operation of the
product exactly, so the outputs may differ by the two scaling forms' last
rounding only: 2^-23 of each value (two half-unit roundings).
"""
import numpy as np
import pytest

import latttmat_gb300 as lt
from cases import seeded_input
from gpu_util import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
oracle = pytest.importorskip("oracle.oracle")


def _product(op, x, dtype, in_place=False):
    xd = torch.tensor(x, device="cuda")
    yd = xd if in_place else torch.empty_like(xd)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    op.perform_op_dev(xd.data_ptr(), yd.data_ptr(), dtype, s.cuda_stream)
    torch.cuda.synchronize()
    return yd.cpu().numpy()


# K = 0.3 and -0.4: scales inside the FP32 range; K = 2.5: past e^60
@pytest.mark.parametrize("L,ec,K", [(12, 0, 0.3), (14, 2, -0.4), (16, 2, 0.3), (18, 0, 2.5)])
def test_reference_order_products(L, ec, K):
    args = ("A", 2, 5, K, 0.6, 0.0, L, 0.0, ec)
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    x = seeded_input(op.rows(), 5)
    y = ref.perform_op(x)
    for in_place in (False, True):
        assert rel_err(_product(op, x, lt.TM_F64, in_place), y) < 1e-12
        assert rel_err(_product(op, x, lt.TM_F64_DF, in_place), y) < 1e-12
        x32 = x.astype(np.float32)
        assert rel_err(_product(op, x32, lt.TM_F32, in_place), ref.perform_op(x32.astype(np.float64))) < 2e-5


def test_reference_order_fp32_scaling_forms():
    op = lt.TMatOp("A", 2, 5, 0.3, 0.6, 0.0, 16, 0.0, 2)
    x = seeded_input(op.rows(), 6).astype(np.float32)
    y = _product(op, x, lt.TM_F32)
    for e in (-60, -90, 60):  # products below 1e-24 and above take the FP64 form
        ys = np.ldexp(_product(op, np.ldexp(x, e), lt.TM_F32).astype(np.float64), -e)
        assert np.all(np.abs(ys - y) <= 2.0 ** -23 * np.abs(y) + 2.0 ** (-126 - e))
    assert np.array_equal(_product(op, np.zeros_like(x), lt.TM_F32), np.zeros_like(x))
    for bad in (np.inf, np.nan):
        xb = x.copy()
        xb[3] = bad
        assert not np.isfinite(_product(op, xb, lt.TM_F32)).any()
    one = np.zeros_like(x)  # all terms of one sign: an infinity stays one
    one[3] = np.inf
    got = _product(op, one, lt.TM_F32)
    assert np.isnan(got).sum() + np.isinf(got).sum() == got.size
