"""The FP64 Gram-Schmidt passes of FGMRES over their row and column ranges:
a solve to 1e-10 must leave that residual for the downloaded matrix (SciPy),
and the Arnoldi estimate it stopped on must agree with the residual formed
from the matrix, which holds as long as the basis is orthonormal to rounding
(estimate and residual differ by at most the loss of orthogonality, near
1e-14, times the condition of the projected problem; 1e-2 of the stop allows
eight orders of it).

Row counts: fewer than one block (n = 3), the 64- and the 256-thread updates
(12, 40), the large passes (190: 323 k rows); restart lengths below, at and above a
column batch, a slice and the default 50, up to the largest (128)."""
import numpy as np
import pytest
import scipy.sparse as sp

import feng_gb300 as fe
from feng_gb300 import kovasznay

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,restart", [(3, 5), (12, 8), (12, 128), (40, 17), (40, 50), (40, 101), (190, 50)])
def test_estimate_and_residual_agree(n, restart):
    _, num, forms = kovasznay.build(n)
    s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(
        precond="amg", precision="fp64", rel_tol=1e-10, restart=restart, max_iter=5000))
    sol = fe.feSolution(s)
    sol.initializeEssentialBC()
    s.setSolution(sol.u)
    s.setToZero()
    s.assembleResiduals()
    s.assembleMatrices()
    st = s.solve()
    ia, ja = s.pattern()
    A, b, x = sp.csr_matrix((s.getMatrix(), ja, ia)), s.getRHS(), s.getDu()
    left = np.linalg.norm(b - A @ x)
    assert left <= 1.01e-10 * np.linalg.norm(b)
    assert st["normAxb"] == pytest.approx(left, rel=1e-2)
