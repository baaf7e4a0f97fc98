"""Products of small operators, whose passes are split by the blocks that they
give and not by what a tile holds: chains from one pass through the widths
where letters move between the passes and chunks shrink, in FP64, FP32 and
double-float, and one-block FP32 products of the reduced Kronecker operators,
against the oracle.

Bars: FP64 and double-float 1e-12 of max|y|, FP32 2e-5 (as the other
products)."""
import numpy as np
import pytest

import latttmat_gb300 as lt
from cases import seeded_input
from gpu_util import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
oracle = pytest.importorskip("oracle.oracle")


def _check(args, dtypes=("f64", "f32", "df")):
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    x = seeded_input(op.rows(), 3)
    y = ref.perform_op(x)
    s = torch.cuda.Stream()
    for name in dtypes:
        dtype, t, bar = {"f64": (lt.TM_F64, torch.float64, 1e-12), "f32": (lt.TM_F32, torch.float32, 2e-5),
                         "df": (lt.TM_F64_DF, torch.float64, 1e-12)}[name]
        xd = torch.tensor(x, dtype=t, device="cuda")
        yd = torch.empty_like(xd)
        torch.cuda.synchronize()
        op.perform_op_dev(xd.data_ptr(), yd.data_ptr(), dtype, s.cuda_stream)
        op.perform_op_dev(xd.data_ptr(), xd.data_ptr(), dtype, s.cuda_stream)
        torch.cuda.synchronize()
        want = y if name != "f32" else ref.perform_op(x.astype(np.float32).astype(np.float64))
        assert rel_err(yd.cpu().numpy(), want) < bar, name
        assert torch.equal(xd, yd), name
    op.close()


@pytest.mark.parametrize("L", [4, 5, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18])
@pytest.mark.parametrize("axialdir", [2, 17, 18, 5])
def test_dnni(axialdir, L):
    _check(("D", 2, axialdir, 0.4, 0.3, 0.1, L, 0.0, 2))


@pytest.mark.parametrize("L", [4, 6, 8, 10, 12, 14, 16, 18])
@pytest.mark.parametrize("axialdir", [3, 7])
def test_bnnni(axialdir, L):
    _check(("B", 2, axialdir, 0.5, 0.6, 0.0, L, 0.2, 0))


@pytest.mark.parametrize("args", [("A", 3, 1, 0.2, 0.4, 0.0, (3, 4), 0.0, 0), ("A", 3, 1, 0.2, 0.4, 0.1, (2, 6), 0.0, 0),
                                  ("A", 2, 5, 0.3, 0.6, 0.0, 11, 0.0, 2), ("A", 2, 5, 0.3, 0.6, 0.0, 13, 0.0, 0),
                                  ("A", 2, 5, -0.3, 0.6, 0.1, 13, 0.0, 2), ("A", 2, 13, 0.4, 0.6, 0.0, 12, 0.0, 2),
                                  ("A", 2, 13, -0.4, 0.6, 0.0, 13, 0.0, 2), ("A", 2, 1, 0.4, 0.6, 0.1, 10, 0.0, 2),
                                  ("A", 2, 1, -0.4, 0.6, 0.1, 11, 0.0, 2)])
def test_kronecker(args):
    _check(args, ("f64", "f32"))
