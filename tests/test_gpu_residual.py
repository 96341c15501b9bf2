"""Taylor-Hood residuals on triangles and tetrahedra against the oracle's node
sums (oracle.taylor_hood), every form present and each one alone, in FP64 and
in the double-float arithmetic of the mixed path.

Sizes: one square or cube of elements up to meshes whose elements leave a
remainder in blocks of 32 elements, and one beyond the 152 x 64 triangles from
which blocks take 64.  Rules: exact to degree 5 and not (degrees 2 to 4), and
the highest tetrahedral degree, whose mixed path is FP64.

Tolerance: sums of at most about 200 terms of one row's elements, each with a
rounding of a few 2^-53 (double-float: 2^-46), relative to the largest entry:
1e-12 leaves a factor of about ten."""
import numpy as np
import pytest

import feng_gb300 as fe
from helpers import rel_err

from oracle.oracle import taylor_hood  # noqa: E402

pytestmark = pytest.mark.gpu

FORMS = {"all": dict(conv=0.9, sigma=-1.0, mu=0.02, divu=1.1, mass=1.3, source=True),
         "conv": dict(conv=-1.0), "stress": dict(sigma=1.0, mu=0.5), "div": dict(divu=-0.7), "mass": dict(mass=2.0),
         "source": dict(divu=1.0, source=True)}
CONST = (0.7, -1.2, 0.4)


def _check(dim, n, degree, precision, which, body=True):
    f = dict(FORMS[which])
    mesh = (fe.Mesh2DP1.generate_square(n, jitter=0.1, seed=3) if dim == 2
            else fe.Mesh3DP1.generate_cube(n, jitter=0.05, seed=4))
    u = fe.createFiniteElementSpace(mesh, fe.VECTOR_LAGRANGE, 2, "U", "Domaine", degree)
    ub = fe.createFiniteElementSpace(mesh, fe.VECTOR_LAGRANGE, 2, "U", "Bord", degree)
    p = fe.createFiniteElementSpace(mesh, fe.LAGRANGE, 1, "P", "Domaine", degree)
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
    source = None
    if f.pop("source", False):
        if body:
            kind, par = (fe.api.SRC_SIN_BODY, (2.5,)) if dim == 2 else (fe.api.SRC_SIN3_BODY, (2.5,))

            def source(*x):
                return (2.5 * np.prod([np.sin(np.pi * c) for c in x], 0),) + (0.0 * x[0],) * (dim - 1)
        else:
            kind, par = fe.api.SRC_CONST_VEC, CONST[:dim]

            def source(*x):
                return tuple(c + 0.0 * x[0] for c in CONST[:dim])
        forms.append(fe.createBilinearForm([u], fe.feSysElm_VectorSource(kind, par)))
    s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(precond="ilu0", precision=precision))
    st = num.setup(0)
    a = mesh.arrays()
    if dim == 2:
        verts = np.stack([a["x"], a["y"]], 1)[a["tri"]]
        quad = np.stack(fe.api.quadrature_rule(degree), 1)
    else:
        verts = np.stack([a["x"], a["y"], a["z"]], 1)[a["tet"]]
        quad = np.stack(fe.api.tet_quadrature_rule(degree), 1)
    rng = np.random.default_rng(7)
    x, xd = rng.uniform(-1, 1, s.nDofs), rng.uniform(-1, 1, s.nDofs)
    s.setSolution(x, xd)
    s.setToZero()
    s.assembleResiduals()
    s.synchronize()
    ia, ja = st.pattern()
    _, rhs = taylor_hood(st.elementDofs(), verts, quad, x, s.nInc, ia, ja, udot=xd, source=source, **f)
    assert rel_err(s.getRHS(), rhs) <= 1e-12


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("which", sorted(FORMS))
@pytest.mark.parametrize("dim", [2, 3])
def test_forms(dim, which, precision):
    _check(dim, 5 if dim == 2 else 3, 5, precision, which, body=which == "all")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dim,n,degree", [(2, 1, 5), (2, 4, 8), (2, 5, 2), (2, 7, 4), (2, 70, 5),
                                          (3, 1, 5), (3, 2, 3), (3, 3, 8), (3, 12, 4)])
def test_sizes_and_rules(dim, n, degree, precision):
    _check(dim, n, degree, precision, "all")
