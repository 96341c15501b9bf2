"""Solver options beside the defaults: the multigrid's smoother degree
(mg_smooth: Chebyshev V-cycles on other operators), inner CG steps (mg_inner)
and the mixed path's Gram-Schmidt variants (gs_passes).

A linear solve to 1e-8 must leave that residual for the downloaded matrix
(SciPy, FP64; 1% for rounding).  In FP64 the preconditioner must also make the
iteration as short as the default does, within half (a smoother of higher degree
only helps, inner CG replaces one V-cycle by at least as good a solve); in mixed
precision counts move by whole restarts, where the FP32 basis loses its
orthogonality."""
import numpy as np
import pytest
import scipy.sparse as sp

import feng_gb300 as fe
from feng_gb300 import cavity, cube, kovasznay
from feng_gb300._lib import FeError
from helpers import problem_spaces

pytestmark = pytest.mark.gpu

CASES = {"flow_2d": lambda: kovasznay.build(40)[1:], "flow_2d_level": lambda: kovasznay.build(6)[1:],
         "scalar_2d": lambda: problem_spaces("diffusion", fe.Mesh2DP1.generate_square(40, jitter=0.1, seed=1)),
         "step_2d": lambda: cavity.build(24, 400.0)[1:], "step_3d": lambda: cube.build(6, 100.0)[1:]}


def _solve(case, precision, **options):
    num, forms = CASES[case]()
    s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(
        precond="amg", precision=precision, rel_tol=1e-8, max_iter=3000, **options))
    sol = fe.feSolution(s)
    sol.initializeEssentialBC()
    if case.startswith("step"):  # a time step's matrix, with its preconditioner
        fe.createTimeIntegrator(fe.BDF2, fe.feNLSolverOptions(), s, sol, 0.0, 1.0, 100)
        s.setTime(0.0, 150.0)
    at = np.arange(s.nDofs)
    s.setSolution(sol.u + 0.01 * np.sin(at) * (at < s.nInc))
    s.setToZero()
    s.assembleResiduals()
    s.assembleMatrices()
    st = s.solve()
    ia, ja = s.pattern()
    A = sp.csr_matrix((s.getMatrix(), ja, ia))
    b = s.getRHS()
    assert np.linalg.norm(b - A @ s.getDu()) <= 1.01e-8 * np.linalg.norm(b)
    return st["nIter"]


@pytest.mark.parametrize("options", [{"mg_smooth": 2}, {"mg_smooth": 4}, {"mg_inner": 1}, {"mg_inner": 3},
                                     {"mg_smooth": 2, "mg_inner": 2}], ids=str)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_multigrid_options(case, precision, options):
    if case == "step_3d" and "mg_inner" in options:  # three components: one V-cycle an application
        with pytest.raises(FeError) as e:
            _solve(case, precision, **options)
        assert e.value.status == -3
        return
    steps = _solve(case, precision, **options)
    if precision == "fp64":
        assert steps <= 1.5 * _solve(case, precision) + 2


@pytest.mark.parametrize("passes", [2, 3])
@pytest.mark.parametrize("case", sorted(CASES))
def test_gram_schmidt_variants(case, passes):
    _solve(case, "mixed", gs_passes=passes)
