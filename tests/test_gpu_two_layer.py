"""Two-layer products and their transposes against the oracle over the widths
where the pass splits and register rounds change, both signs of the couplings,
flip on and off, in place.  Bar: 1e-12 of max|y| (FP64, as the other products).
"""
import numpy as np
import pytest

import latttmat_gb300 as lt
from cases import seeded_input
from gpu_util import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
oracle = pytest.importorskip("oracle.oracle")


def _run(op, x):
    xd = torch.tensor(x, device="cuda")
    yd = torch.empty_like(xd)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    op.perform_op_dev(xd.data_ptr(), yd.data_ptr(), lt.TM_F64, s.cuda_stream)
    op.perform_op_dev(xd.data_ptr(), xd.data_ptr(), lt.TM_F64, s.cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(xd, yd)
    return yd.cpu().numpy()


@pytest.mark.parametrize("model,ax,L,ec,K,k,h", [
    ("A", 2, 4, 0, 0.5, 0.3, 0.0), ("A", 2, 5, 0, -0.4, 0.3, 0.1), ("A", 2, 8, 0, 0.4, 0.6, 0.1),
    ("A", 2, 9, 0, 0.4, 0.6, 0.0), ("A", 2, 10, 0, 0.3, -0.2, 0.05),
    ("A", 0, 4, 0, 0.5, 0.3, 0.0), ("A", 0, 6, 0, -0.4, 0.3, 0.1), ("A", 0, 7, 0, 0.4, 0.6, 0.1),
    ("A", 0, 10, 0, 0.3, 0.6, 0.0),
    ("A", 6, 5, 0, 0.4, 0.6, 0.0), ("A", 6, 8, 2, -0.4, 0.6, 0.0), ("A", 6, 9, 0, 0.4, 0.6, 0.1),
    ("A", 6, 11, 2, 0.3, 0.6, 0.0), ("B", 6, 6, 0, 0.5, 0.4, 0.0), ("B", 6, 10, 2, 0.4, -0.3, 0.0),
])
def test_two_layer(model, ax, L, ec, K, k, h):
    args = (model, 2, ax, K, k, h, L, 0.2 if model == "B" else 0.0, ec)
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    assert op.rows() == ref.n
    x = seeded_input(op.rows(), 6)
    assert rel_err(_run(op, x), ref.perform_op(x)) < 1e-12
    if ax != 0:
        assert rel_err(_run(op.get_t_instance(), x), ref.perform_op_t(x)) < 1e-12
