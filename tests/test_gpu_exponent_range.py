"""Products whose sums would leave the exponent range before their factors
bring them back: FP32 and double-float chains whose weights come near the end
of the FP32 range; and a strongly frustrated point whose values lie far below
the largest step, where nothing may be scaled down.

Bars: double-float 1e-12 of max|y|, FP32 2e-5 (as the other products)."""
import numpy as np
import pytest

import latttmat_gb300 as lt
from cases import seeded_input
from gpu_util import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
oracle = pytest.importorskip("oracle.oracle")

TYPES = {"f32": (lt.TM_F32, np.float32, 2e-5), "df": (lt.TM_F64_DF, np.float64, 1e-12)}


@pytest.mark.parametrize("args,types", [
    (("D", 2, 18, 8.0, 2.0, 0.0, 12, 0.0, 2), ("f32", "df")), (("D", 2, 18, 12.0, 1.0, 0.2, 12, 0.0, 2), ("f32",)),
    (("D", 2, 17, 8.0, 2.0, 0.2, 11, 0.0, 2), ("f32", "df")), (("D", 2, 18, 8.0, 2.0, 0.0, 8, 0.0, 2), ("f32", "df")),
    (("B", 2, 3, -3.0, -1.0, 0.0, 12, 0.3, 2), ("df",)), (("B", 2, 7, -3.0, -1.0, 0.2, 12, 0.3, 2), ("df",)),
    (("D", 2, 5, 2.0, 2.0, 0.0, 13, 0.0, 2), ("f32",)), (("B", 2, 7, 2.0, 2.0, 0.0, 12, 0.3, 2), ("f32",))])
def test_products(args, types):
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    s = torch.cuda.Stream()
    for name in types:
        dtype, kind, bar = TYPES[name]
        x = seeded_input(op.rows(), 9).astype(kind)
        want = ref.perform_op(x.astype(np.float64))
        xd = torch.tensor(x, device="cuda")
        yd = torch.empty_like(xd)
        torch.cuda.synchronize()
        op.perform_op_dev(xd.data_ptr(), yd.data_ptr(), dtype, s.cuda_stream)
        torch.cuda.synchronize()
        got = yd.double().cpu().numpy()
        assert np.isfinite(got).all() and rel_err(got, want) < bar, name
