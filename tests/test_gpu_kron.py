"""Kronecker-core products against the oracle: tile passes of the full
x-ANNNI operator at the widths where the pass rule changes, and prefix-tree
products of the reduced operators (odd widths, 3D layers) from the smallest
tree up, both signs of betaJ, flip on and off, in place.

Bars: FP64 1e-12 of max|y|, FP32 2e-5 of max|y| (as the other products).
"""
import numpy as np
import pytest

import latttmat_gb300 as lt
from cases import seeded_input
from gpu_util import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
oracle = pytest.importorskip("oracle.oracle")


def _check(args, seed=3):
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    assert op.rows() == ref.n
    x = seeded_input(op.rows(), seed)
    y = ref.perform_op(x)
    s = torch.cuda.Stream()
    for dtype, t, bar in ((lt.TM_F64, torch.float64, 1e-12), (lt.TM_F32, torch.float32, 2e-5)):
        xd = torch.tensor(x, dtype=t, device="cuda")
        yd = torch.empty_like(xd)
        torch.cuda.synchronize()
        op.perform_op_dev(xd.data_ptr(), yd.data_ptr(), dtype, s.cuda_stream)
        op.perform_op_dev(xd.data_ptr(), xd.data_ptr(), dtype, s.cuda_stream)
        torch.cuda.synchronize()
        want = y if t is torch.float64 else ref.perform_op(x.astype(np.float32).astype(np.float64))
        assert rel_err(yd.cpu().numpy(), want) < bar
        assert torch.equal(xd, yd)
    op.close()


@pytest.mark.parametrize("L,K", [(4, 0.5), (5, -0.6), (9, 0.5), (10, 0.4), (11, -0.3), (15, 0.4), (18, 0.3), (19, 0.7),
                                 (20, 0.3), (21, 0.3)])
def test_full_tile_passes(L, K):
    _check(("A", 2, 1, K, 0.4, 0.1, L, 0.0, 0))


def test_full_fp32_scaling_outside_fp32_range():
    # weights past 2^90 and below 2^-70: the FP64 form of the scaling
    _check(("A", 2, 1, 4.5, 0.9, 0.3, 16, 0.0, 0))


@pytest.mark.parametrize("L,ec,K,h", [(4, 2, 0.5, 0.0), (5, 0, 0.4, 0.0), (7, 2, -0.5, 0.0), (8, 0, 0.5, 0.0),
                                      (9, 0, 0.3, 0.1), (13, 2, 0.3, 0.0), (17, 0, -0.4, 0.0), (19, 2, 0.3, 0.0)])
def test_tree_2d(L, ec, K, h):
    _check(("A", 2, 5, K, 0.6, h, L, 0.0, ec))


@pytest.mark.parametrize("size,k,h", [((2, 2), 0.3, 0.0), ((2, 3), 0.0, 0.1), ((3, 3), 0.0, 0.0), ((3, 4), 0.5, 0.1),
                                      ((4, 4), 0.0, 0.0), ((3, 6), 0.4, 0.0), ((5, 4), 0.4, 0.0)])
def test_tree_3d(size, k, h):
    _check(("A", 3, 1, 0.25, k, h, size, 0.0, 0))


@pytest.mark.parametrize("L,ec", [(12, 2), (13, 0), (10, 0)])
def test_open_boundary_full_space(L, ec):
    _check(("A", 2, 13, 0.4, 0.6, 0.0, L, 0.0, ec))
