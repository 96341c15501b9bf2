"""The degree-1 V-cycle on its combined level operators (T, Q, Q^T: two
kernels per level), through the preconditioner application z = B r / s, by
the properties that a V-cycle with the same damped Jacobi step before and
after the coarse correction has (B symmetric; the error operator I - B K
symmetric in the K inner product with spectrum in [0, 1): a product S C S of
the smoother and a K-orthogonal projection or its approximation), which a
wrong entry, weight or row of T, Q or Q^T breaks.  (The hierarchy itself cannot
be restated bit for bit: the P2 stiffness ties the strongest connections of
every edge node, which rounding decides.)

Sizes: a single level (8: B = K^-1), two levels in CSR (20), the smallest
finest level in sliced ELL with a ragged last slice (37), a larger one (64).
Tolerances: symmetry and the lower end of the spectrum 1e-10 (FP64 rounding
times the condition of the coarsest operator, about 1e4); FP32 against FP64
5e-5 of max |z| (row sums of up to 150 terms at 6e-8 each on every level)."""
import sys

import numpy as np
import pytest
import scipy.sparse as sp

import feng_gb300 as fe
from conftest import ROOT
from feng_gb300 import kovasznay
from helpers import problem_spaces

sys.path.insert(0, str(ROOT / "oracle"))
import newton_oracle as no  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 20, 37, 64])
@pytest.mark.parametrize("problem", ["diffusion", "ns"])
def test_vcycle_properties(problem, n):
    if problem == "ns":
        pb = no.Problem2D("ns_kovasznay", n, re=40.0, seed=3)
        _, num, forms = kovasznay.build(n, 40.0, seed=3)
    else:
        pb = no.Problem2D("diffusion", n, seed=3)
        num, forms = problem_spaces("diffusion", fe.Mesh2DP1.generate_square(n, jitter=0.1, seed=3))
    rng = np.random.default_rng(n)
    systems = {}
    for precision in ("fp64", "mixed"):
        s_ = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(precond="amg", precision=precision))
        s_.setSolution(pb.u_bc)
        s_.setToZero()
        s_.assembleMatrices()
        systems[precision] = s_
    Kia, Kja, Ka = pb.K
    K = sp.csr_matrix((Ka, Kja, Kia))
    J = sp.csr_matrix((pb.matrix(pb.u_bc, 4), pb.keep["ja"], pb.keep["ia"]))
    s = J.diagonal()[pb.dofx].sum() / K.diagonal().sum()
    comps = [pb.dofx] + ([pb.dofy] if problem == "ns" else [])

    def apply(precision, v, c):
        """B v on component c (no pressure part: z_p = 0)."""
        r = np.zeros(pb.n_inc)
        r[comps[c]] = v
        z = systems[precision].applyPreconditioner(r)
        assert np.max(np.abs(np.delete(z, comps[c])), initial=0.0) <= 1e-14 * np.max(np.abs(z))
        return s * z[comps[c]]

    m = K.shape[0]
    grid = np.arange(m) / m
    vectors = [rng.uniform(-1, 1, m), np.sin(np.pi * grid), np.ones(m), np.eye(1, m, m // 2)[0], np.eye(1, m, m - 1)[0]]
    for c in range(len(comps)):
        b = [apply("fp64", v, c) for v in vectors]
        for i in range(len(vectors)):
            for j in range(i):
                scale = np.linalg.norm(b[i]) * np.linalg.norm(vectors[j])
                assert abs(b[i] @ vectors[j] - b[j] @ vectors[i]) <= 1e-10 * scale
        for v, bv in zip(vectors, b):
            zf = apply("mixed", v, c)
            assert np.max(np.abs(zf - bv)) <= 5e-5 * np.max(np.abs(bv))
        for e in vectors:
            for _ in range(6):  # power steps of I - B K
                d = e - apply("fp64", K @ e, c)
                q = (e @ (K @ d)) / (e @ (K @ e))
                assert -1e-10 <= q < 0.95
                if n == 8:
                    assert np.max(np.abs(d)) <= 1e-10 * np.max(np.abs(e))
                    break
                e = d
