"""The block-column copy of the matrix that the solves multiply with from
75,000 rows on, against the CSR matrix: a solve to 1e-6 must leave that
residual for the downloaded matrix (SciPy, FP64), which needs right products
in the iteration and right residuals at its restarts.

Cases: node blocks of two and three unknowns, two-unknown blocks at odd
columns (an odd number of pressures numbered first), no blocks (scalar P2 on
triangles and tetrahedra); pressure rows and columns are single.  Tolerance:
the FP64 solve stops on the Arnoldi estimate, the mixed one on the residual of
the FP32 matrix with rounding near 1e-13, both within 1% of the stop."""
import numpy as np
import pytest
import scipy.sparse as sp

import feng_gb300 as fe
from feng_gb300 import cavity, cube, exact, kovasznay
from helpers import problem_spaces

pytestmark = pytest.mark.gpu


def _odd_blocks(n):
    m = fe.Mesh2DP1.generate_square(n, *kovasznay.DOMAIN, jitter=0.1, seed=1)
    uex, pex = exact.kovasznay_velocity(40.0), exact.kovasznay_pressure(40.0)
    p = fe.createFiniteElementSpace(m, fe.LAGRANGE, 1, "P", "Domaine", 8, pex)
    pp = fe.createFiniteElementSpace(m, fe.LAGRANGE, 1, "P", "PointPression", 8, pex)
    u = fe.createFiniteElementSpace(m, fe.VECTOR_LAGRANGE, 2, "U", "Domaine", 8, uex)
    ub = fe.createFiniteElementSpace(m, fe.VECTOR_LAGRANGE, 2, "U", "Bord", 8, uex)
    num = fe.feMetaNumber(m, [p, pp, u, ub], [pp, ub])
    return num, [fe.createBilinearForm([u], fe.feSysElm_VectorConvectiveAcceleration(-1.0)),
                 fe.createBilinearForm([p, u], fe.feSysElm_MixedDivergence(1.0)),
                 fe.createBilinearForm([u, p], fe.feSysElm_DivergenceNewtonianStress(1.0, 1 / 40.0))]


def _tet_diffusion(n):
    m = fe.Mesh3DP1.generate_cube(n, jitter=0.05, seed=1)
    u = fe.createFiniteElementSpace(m, fe.LAGRANGE, 2, "U", "Domaine", 4)
    ub = fe.createFiniteElementSpace(m, fe.LAGRANGE, 2, "U", "Bord", 4)
    num = fe.feMetaNumber(m, [u, ub], [ub])
    return num, [fe.createBilinearForm([u], fe.feSysElm_Diffusion(1.0)),
                 fe.createBilinearForm([u], fe.feSysElm_Source(fe.api.SRC_SIN3, (1.0,)))]


CASES = {"flow_2d": lambda: kovasznay.build(97)[1:], "flow_2d_odd": lambda: _odd_blocks(101),
         "flow_3d": lambda: cube.build(16, 100.0)[1:], "scalar_2d": lambda: problem_spaces(
             "diffusion", fe.Mesh2DP1.generate_square(140, jitter=0.1, seed=1)), "scalar_3d": lambda: _tet_diffusion(22)}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_solve_leaves_the_asked_residual(case, precision):
    num, forms = CASES[case]()
    krylov = "cg" if case.startswith("scalar") and precision == "fp64" else "fgmres"
    s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(
        krylov=krylov, precond="amg", precision=precision, rel_tol=1e-6, max_iter=2000))
    assert s.nInc >= 75000
    sol = fe.feSolution(s)
    sol.initializeEssentialBC()
    if case == "flow_3d":  # a time step's matrix, with its preconditioner
        fe.createTimeIntegrator(fe.BDF2, fe.feNLSolverOptions(), s, sol, 0.0, 1.0, 100)
        s.setTime(0.0, 150.0)
    s.setSolution(sol.u + 0.01 * np.sin(np.arange(s.nDofs)) * (np.arange(s.nDofs) < s.nInc))
    s.setToZero()
    s.assembleResiduals()
    s.assembleMatrices()
    st = s.solve()
    ia, ja = s.pattern()
    A = sp.csr_matrix((s.getMatrix(), ja, ia))
    b, x = s.getRHS(), s.getDu()
    left = np.linalg.norm(b - A @ x)
    assert st["nIter"] > 3
    assert left <= 1.01e-6 * np.linalg.norm(b)
    # the reported residual: the recurrence's (CG) or the one at the end
    assert st["normAxb"] == pytest.approx(left, rel=1e-2)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_product_matches_rows(case, precision):
    """The iteration's product itself, row by row: a sum of k products of rounded
    operands is off by at most (k + 2) roundings of the sum of their magnitudes."""
    num, forms = CASES[case]()
    s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(precond="none", precision=precision))
    assert s.nInc >= 75000
    rng = np.random.default_rng(5)
    s.setSolution(rng.uniform(-1, 1, s.nDofs))
    s.setTime(0.0, 150.0)
    s.setToZero()
    s.assembleMatrices()
    ia, ja = s.pattern()
    A = sp.csr_matrix((s.getMatrix(), ja, ia))
    x = rng.uniform(-1, 1, s.nInc)
    y = s.applyMatrix(x)
    unit = 2.0 ** (-53 if precision == "fp64" else -24)
    assert np.all(np.abs(y - A @ x) <= (np.diff(ia) + 2) * unit * (abs(A) @ np.abs(x)))
    s.setMatrixToZero()  # the copy follows the matrix
    assert np.all(s.applyMatrix(x) == 0.0)
