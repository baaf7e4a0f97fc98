"""Even/odd products at the widths where the tiles of the 8-byte types are
first split over two (L = 26) and four (L = 28) CTAs, and the FP32 tile is
whole, in all three precisions against the oracle.

Bars: FP64 and double-float 1e-12 of max|y|, FP32 2e-5 (the bars of the
other product tests)."""
import numpy as np
import pytest

import latttmat_gb300 as lt

pytestmark = pytest.mark.gpu
oracle = pytest.importorskip("oracle.oracle")
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("L,bj,h", [(26, 0.35, 0.0), (26, -0.3, 0.05), (28, -0.25, 0.0)])
def test_products(L, bj, h):
    args = ("A", 2, 5, bj, 0.5, h, L, 0.0, 0)
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    x = np.random.default_rng(L).standard_normal(op.rows())
    yr = ref.perform_op(x)
    stream = torch.cuda.current_stream().cuda_stream
    for dt, tdt, bar in ((lt.TM_F32, torch.float32, 2e-5), (lt.TM_F64_DF, torch.float64, 1e-12),
                         (lt.TM_F64, torch.float64, 1e-12)):
        xd = torch.tensor(x, dtype=tdt, device="cuda")
        yd = torch.empty_like(xd)
        op.perform_op_dev(xd.data_ptr(), yd.data_ptr(), dt, stream)
        torch.cuda.synchronize()
        err = np.max(np.abs(yd.cpu().numpy().astype(np.float64) - yr)) / np.max(np.abs(yr))
        assert err < bar, (dt, err)
