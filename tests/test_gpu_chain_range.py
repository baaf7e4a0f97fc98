"""FP32 chain products whose values leave the FP32 exponent range: sums of
carried letters with an infinity stay infinite (all weights are positive), as
in FP64, and do not become NaN.
"""
import numpy as np
import pytest

import latttmat_gb300 as lt

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

OPS = [("D", 2, 2, 0.4, 0.3, 0.1, 9, 0.0, 2), ("D", 2, 2, 0.4, 0.3, 0.1, 15, 0.0, 2),
       ("D", 2, 18, 0.4, 0.3, 0.1, 14, 0.0, 2), ("D", 2, 5, 0.4, 0.3, 0.0, 13, 0.0, 2),
       ("B", 2, 3, 0.5, 0.6, 0.0, 8, 0.2, 2), ("B", 2, 7, 0.5, 0.6, 0.0, 12, 0.2, 2)]


def _product(op, x):
    xd = torch.tensor(x, device="cuda")
    yd = torch.empty_like(xd)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    op.perform_op_dev(xd.data_ptr(), yd.data_ptr(), lt.TM_F32, s.cuda_stream)
    torch.cuda.synchronize()
    return yd.cpu().numpy()


@pytest.mark.parametrize("args", OPS)
def test_infinite_sums(args):
    op = lt.TMatOp(*args)
    n = op.rows()
    x = np.zeros(n, dtype=np.float32)
    x[n // 3] = np.inf
    assert np.all(np.isposinf(_product(op, x)))
    x[n // 3] = -np.inf
    assert np.all(np.isneginf(_product(op, x)))
    x[n // 3] = np.nan
    assert np.all(np.isnan(_product(op, x)))
    x[:] = 3e38  # overflows in the input weights or on the way
    y = _product(op, x)
    assert not np.isnan(y).any() and np.isposinf(y).any()
