"""Solves around the sizes of the short Gram-Schmidt step (one element per
thread, up to 262144 rows): one block, a partial last block, the most rows it
takes and the first it does not, wide subspaces (more than eight and sixteen
columns), symmetric and general operators.

Bars: eigenvalues within 1e-10 of the oracle's; ||T v - lambda v|| / |lambda|
at most 1e-10 (tol 1e-12, the product's own error below 1e-12 of max|y|).
"""
import numpy as np
import pytest

import latttmat_gb300 as lt

pytestmark = pytest.mark.gpu
oracle = pytest.importorskip("oracle.oracle")


@pytest.mark.parametrize("args,nev,ncv", [
    (("A", 2, 1, 0.6, 0.2, 0.05, 7, 0.0, 0), 2, 0), (("A", 2, 5, 0.4, 0.3, 0.05, 13, 0.0, 0), 3, 20),
    (("A", 2, 1, 0.6, 0.2, 0.05, 18, 0.0, 0), 2, 12), (("A", 2, 1, 0.6, 0.2, 0.05, 19, 0.0, 0), 2, 12),
    (("D", 2, 5, 0.4, 0.3, 0.0, 14, 0.0, 0), 2, 0), (("B", 2, 7, 0.4, 0.3, 0.0, 12, 0.0, 0), 2, 18),
    (("A", 2, 2, 0.4, 0.3, 0.0, 6, 0.0, 0), 2, 0), (("A", 2, 6, 0.4, 0.3, 0.05, 7, 0.0, 0), 2, 9),
])
def test_solves(args, nev, ncv):
    op, ref = lt.TMatOp(*args), oracle.OracleOp(*args)
    vals, vecs, _, info = op.eigs(nev, ncv=ncv, tol=1e-12, vectors=True)
    want = ref.eigs(nev)
    np.testing.assert_allclose(np.sort(np.abs(vals))[::-1], np.sort(np.abs(want))[::-1], rtol=1e-10)
    nf = op.getnormfactor()
    for i in range(nev):
        v = vecs[i]
        tv = ref.perform_op(np.ascontiguousarray(v.real))
        if np.iscomplexobj(v):
            tv = tv + 1j * ref.perform_op(np.ascontiguousarray(v.imag))
        lam = vals[i] * nf
        assert np.linalg.norm(tv - lam * v) <= 1e-10 * abs(lam) * np.linalg.norm(v)
    assert info["nconv"] == nev
