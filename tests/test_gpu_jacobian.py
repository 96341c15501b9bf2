"""The Taylor-Hood Jacobian from element matrices and a colored scatter (the
FP64 path, and FP32 where a row is too long for the row-owned kernel) against
the oracle.

Sizes: element counts below, at and beside a block's 32, a fan of 60 triangles
around a vertex (rows of 417 entries, one element a color), and more elements
than the 2^18 that the buffer holds at a time.  Tolerance: relative to the
largest entry, FP64 sums of a few hundred roundings of 2^-53 at most (1e-12
leaves a factor of ten), FP32 ones 1e-5 likewise."""
import numpy as np
import pytest

import feng_gb300 as fe
from helpers import element_xy, rel_err

from oracle.oracle import OracleProblem, taylor_hood  # noqa: E402

pytestmark = pytest.mark.gpu

FORMS = {"all": dict(conv=0.9, sigma=-1.0, mu=0.02, divu=1.1, mass=1.3), "conv": dict(conv=-1.0),
         "stress": dict(sigma=1.0, mu=0.5), "div": dict(divu=-0.7), "mass": dict(mass=2.0)}


def _system(mesh, f, precision):
    u = fe.createFiniteElementSpace(mesh, fe.VECTOR_LAGRANGE, 2, "U", "Domaine", 5)
    ub = fe.createFiniteElementSpace(mesh, fe.VECTOR_LAGRANGE, 2, "U", "Bord", 5)
    p = fe.createFiniteElementSpace(mesh, fe.LAGRANGE, 1, "P", "Domaine", 5)
    num = fe.feMetaNumber(mesh, [u, ub, p], [ub])
    forms = []
    if "mass" in f:
        forms.append(fe.createBilinearForm([u], fe.feSysElm_TransientVectorMass(f["mass"])))
    if "conv" in f:
        forms.append(fe.createBilinearForm([u], fe.feSysElm_VectorConvectiveAcceleration(f["conv"])))
    if "divu" in f:
        forms.append(fe.createBilinearForm([p, u], fe.feSysElm_MixedDivergence(f["divu"])))
    if "sigma" in f:
        forms.append(fe.createBilinearForm([u, p], fe.feSysElm_DivergenceNewtonianStress(f["sigma"], f["mu"])))
    s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(precond="ilu0", precision=precision))
    x = np.random.default_rng(3).uniform(-1, 1, s.nDofs)
    s.setSolution(x, np.zeros(s.nDofs))
    s.setTime(0.0, 1.7)
    s.setToZero()
    s.assembleMatrices()
    return num, forms, s, x


def _fan(m):
    t = 2 * np.pi * np.arange(m) / m
    k = np.arange(m)
    tri = np.stack([np.zeros(m, int), 1 + k, 1 + (k + 1) % m], 1)
    return fe.Mesh2DP1.from_arrays(np.concatenate([[0.1], np.cos(t)]), np.concatenate([[0.05], np.sin(t)]), tri,
                                   np.array([[1, 2]]))


def _check(mesh, f, precision, tol):
    num, _, s, x = _system(mesh, f, precision)
    st, a = num.setup(0), mesh.arrays()
    verts = np.stack([a["x"], a["y"]], 1)[a["tri"]]
    ia, ja = st.pattern()
    vals, _ = taylor_hood(st.elementDofs(), verts, np.stack(fe.api.quadrature_rule(5), 1), x, s.nInc, ia, ja,
                          udot=np.zeros(s.nDofs), c0=1.7, **f)
    assert s.jacobianRoute == 0
    assert rel_err(s.getMatrix(), vals) <= tol


@pytest.mark.parametrize("n,which", [(1, "all"), (4, "all"), (5, "all")] + [(5, w) for w in sorted(FORMS) if w != "all"])
def test_square(n, which):
    _check(fe.Mesh2DP1.generate_square(n, jitter=0.1, seed=3), FORMS[which], "fp64", 1e-12)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
def test_fan(precision, tol):
    _check(_fan(60), FORMS["all"], precision, tol)


def test_more_elements_than_the_buffer():
    mesh = fe.Mesh2DP1.generate_square(363, jitter=0.1, seed=3)
    num, forms, s, x = _system(mesh, FORMS["all"], "fp64")
    st = num.setup(0)
    off, el = st.coloring()
    ia, ja = st.pattern()
    op = OracleProblem(2, st.elementDofs(), element_xy(mesh), s.nInc, s.nDofs, off, el, ia, ja,
                       fe.api.quadrature_rule(5), [b.sysElm for b in forms])
    assert rel_err(s.getMatrix(), op.matrix(x, 1.7)) <= 1e-12
