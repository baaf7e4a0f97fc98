"""Chain products (DNNI, diagonal BNNNI) against the oracle at the edges of the
pass plan: the smallest rings (one pass), widths where a second and a third
pass appear, every tile size the tuning table takes, open boundaries, flip on
and off, negative couplings, transposes, in place.

Bars: FP64 and double-float 1e-12 of max|y|, FP32 2e-5 (as the other products).
"""
import numpy as np
import pytest

import latttmat_gb300 as lt
from cases import seeded_input
from gpu_util import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
oracle = pytest.importorskip("oracle.oracle")
BARS = ((lt.TM_F64, torch.float64, 1e-12), (lt.TM_F64_DF, torch.float64, 1e-12), (lt.TM_F32, torch.float32, 2e-5))


def _run(op, x, dtype, t):
    xd = torch.tensor(x, dtype=t, device="cuda")
    yd = torch.empty_like(xd)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    op.perform_op_dev(xd.data_ptr(), yd.data_ptr(), dtype, s.cuda_stream)
    op.perform_op_dev(xd.data_ptr(), xd.data_ptr(), dtype, s.cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(xd, yd)
    return yd.cpu().numpy()


def _check(args, bars=BARS):
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    assert op.rows() == ref.n
    x = seeded_input(op.rows(), 4)
    y, yt = ref.perform_op(x), None
    for dtype, t, bar in bars:
        assert rel_err(_run(op, x, dtype, t), y) < bar
    if args[0] == "B":
        yt = ref.perform_op_t(x)
        tr = op.get_t_instance()
        for dtype, t, bar in bars:
            assert rel_err(_run(tr, x, dtype, t), yt) < bar


@pytest.mark.parametrize("ax,ec,h", [(1, 0, 0.1), (17, 0, 0.1), (18, 0, 0.0), (5, 2, 0.0), (5, 0, 0.0)])
@pytest.mark.parametrize("L,K", [(4, 0.5), (5, -0.4), (9, 0.3), (12, 0.4), (13, -0.5), (15, 0.4)])
def test_dnni(L, K, ax, ec, h):
    if L == 4 and ax == 5:
        K = 0.45
    _check(("D", 2, ax, K, 0.35, h, L, 0.0, ec))


@pytest.mark.parametrize("ax,ec,h", [(3, 0, 0.1), (7, 2, 0.0), (7, 0, 0.0)])
@pytest.mark.parametrize("L,K", [(4, 0.5), (6, -0.4), (10, 0.3), (12, 0.4), (14, -0.5), (16, 0.4)])
def test_bnnni(L, K, ax, ec, h):
    _check(("B", 2, ax, K, 0.6, h, L, 0.2, ec))


@pytest.mark.parametrize("model,ax,L", [("D", 5, 17), ("D", 1, 16), ("B", 7, 16), ("B", 3, 14)])
def test_tile_sizes(model, ax, L):
    args = (model, 2, ax, 0.4, 0.3, 0.0, L, 0.1 if model == "B" else 0.0, 2)
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    x = seeded_input(op.rows(), 5)
    y = ref.perform_op(x)
    try:
        for dtype, t, bar in BARS:
            for tile in range(10, 15 if dtype == lt.TM_F32 else 14):
                for threads in (64, 128, 256):
                    lt.chain_set_tuning(model, L, dtype, tile, threads)
                    assert rel_err(_run(op, x, dtype, t), y) < bar
    finally:
        for dtype in (lt.TM_F32, lt.TM_F64_DF):
            lt.chain_set_tuning(model, L, dtype, 0, 0)
