"""FP64 products of the second two-layer operator (a 4 x 4 factor on every bit
pair): large betaJ, where the pair steps' sums would leave the FP64 range
before the output factor brings them back, and ratios on either side of one.

Bar: 1e-12 of max|y| (as the other products)."""
import numpy as np
import pytest

import latttmat_gb300 as lt
from cases import seeded_input
from gpu_util import rel_err

pytestmark = pytest.mark.gpu
oracle = pytest.importorskip("oracle.oracle")


@pytest.mark.parametrize("args", [
    ("A", 2, 0, 20.0, 2.0, 0.2, 6, 0.0, 2),
    ("A", 2, 0, 40.0, 0.5, 0.0, 6, 0.0, 2),
    ("A", 2, 0, 20.0, -1.0, 0.0, 6, 0.0, 2),
    ("A", 2, 0, 15.0, -2.5, 0.0, 6, 0.0, 2),
    ("A", 2, 0, -0.4, 0.3, 0.1, 5, 0.0, 2),
    ("A", 2, 0, 0.4, -0.3, 0.1, 6, 0.0, 2),
    ("A", 2, 0, -0.4, -1.5, 0.1, 6, 0.0, 2),
    ("A", 2, 0, 0.4, 1.5, 0.0, 7, 0.0, 2),
    ("A", 2, 0, 0.4, -1.5, 0.0, 6, 0.0, 2),
    ("A", 2, 0, -0.4, 1.5, 0.0, 6, 0.0, 2)])
def test_products(args):
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    x = seeded_input(op.rows(), 9)
    got = op.perform_op(x)
    assert np.isfinite(got).all() and rel_err(got, ref.perform_op(x)) < 1e-12
