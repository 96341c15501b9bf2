"""The level-scheduled ILU(0) preconditioner on the device against the
oracle's serial ILU(0) (Saad, Alg. 10.4, oracle/fe_oracle.c), through the
C ABI (fe_cuda_apply_preconditioner).

The device factorisation applies each row's updates in the serial order, so
its factors equal the serial ones; the triangular solves sum each row in a
different order.  Tolerance of z = (LU)^-1 r: 1e-12 relative to max |z| in
FP64, 1e-5 with the FP32 factors of the mixed path.  Cases: the 64 x 64 P2
diffusion system of the CPU-runnable configuration as one block (254
levels in its L and in its U part), and a Taylor-Hood Jacobian in
block-Jacobi form (the blocks of the set-up's partition)."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import feng_gb300 as fe
from conftest import ROOT, load_golden
from helpers import golden_mesh, problem_spaces

from oracle.oracle import OracleProblem  # noqa: E402

pytestmark = pytest.mark.gpu


def _oracle_ilu(g, vals, r, blocks=None):
    from feng_gb300.api import quadrature_rule
    nloc = g["adr"].size // len(g["tri"])
    op = OracleProblem(1 if nloc == 6 else 2, g["adr"], np.zeros((len(g["tri"]), 6)), int(g["nInc"]),
                       int(g["nDofs"]), g["color_offsets"], g["color_elements"], g["ia"], g["ja"],
                       quadrature_rule(int(g["quad_degree"])), [])
    return op.apply_ilu(vals, r, blocks)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_ilu0_single_block_matches_serial(precision):
    g = load_golden("diffusion_p2_64")
    num, forms = problem_spaces("diffusion", golden_mesh(g))
    sys_ = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(krylov="fgmres", precond="ilu0",
                                                                            precision=precision))
    sys_.setSolution(g["u0"])
    sys_.setToZero()
    sys_.assembleMatrices()
    r = np.random.default_rng(3).uniform(-1, 1, sys_.nInc)
    z = sys_.applyPreconditioner(r)
    zo = _oracle_ilu(g, sys_.getMatrix(), r)
    tol = 1e-12 if precision == "fp64" else 1e-5
    assert np.max(np.abs(z - zo)) <= tol * np.max(np.abs(zo))


def test_ilu0_block_jacobi_matches_serial():
    g = load_golden("kovasznay_th_8")
    num, forms = problem_spaces("ns_kovasznay", golden_mesh(g), 40.0)
    opts = fe.LinearSolverOptions(precond="bjacobi-ilu0", pc_block_rows=64)
    sys_ = fe.createLinearSystem(fe.CUDA, forms, num, opts)
    sys_.setSolution(g["u0"])
    sys_.setToZero()
    sys_.assembleMatrices()
    r = np.random.default_rng(4).uniform(-1, 1, sys_.nInc)
    z = sys_.applyPreconditioner(r)
    zo = _oracle_ilu(g, sys_.getMatrix(), r, num.setup(64).blocks())
    assert np.max(np.abs(z - zo)) <= 1e-12 * np.max(np.abs(zo))


def _ilu_reference(A, r, blocks):
    """(LU)^-1 r of the ILU(0) of A restricted to the diagonal blocks (Saad,
    Alg. 10.4), row by row in FP64."""
    n = len(r)
    rows = []
    for i in range(n):
        c, v = A.indices[A.indptr[i]:A.indptr[i + 1]], A.data[A.indptr[i]:A.indptr[i + 1]]
        keep = blocks[c] == blocks[i]
        rows.append(dict(zip(c[keep].tolist(), v[keep].tolist())))
    for i in range(n):
        for k in sorted(c for c in rows[i] if c < i):
            rows[i][k] /= rows[k][k]
            for j, u in rows[k].items():
                if j > k and j in rows[i]:
                    rows[i][j] -= rows[i][k] * u
    z = r.copy()
    for i in range(n):
        z[i] -= sum(v * z[c] for c, v in rows[i].items() if c < i)
    for i in range(n - 1, -1, -1):
        z[i] = (z[i] - sum(v * z[c] for c, v in rows[i].items() if c > i)) / rows[i][i]
    return z


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,rows", [(1, 0), (6, 0), (9, 1), (9, 40), (14, 0), (40, 256)])
def test_ilu0_solves_match_serial_over_block_shapes(n, rows, precision):
    """One block and many (the smallest partition up to 256 rows), levels of
    one row and of more rows than a step, rows longer than a step's entries (the flow's
    vertex rows): the solves with the vector in shared memory.  The flow's
    pressure rows have no diagonal entry of their own: their pivots come from
    the elimination.  Tolerances:
    rounding times the growth of that elimination, taken as 1e4 for the
    mass-dominated velocity block (1e-11 and 1e-2 of max |z|)."""
    import scipy.sparse as sp
    mesh = fe.Mesh2DP1.generate_square(n, jitter=0.1, seed=2)
    num, forms = problem_spaces("ns_cavity_bdf2" if n < 40 else "diffusion", mesh, 40.0)
    sys_ = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(
        krylov="fgmres", precond="ilu0" if rows == 0 else "bjacobi-ilu0", pc_block_rows=max(rows, 1),
        precision=precision))
    sys_.setSolution(np.random.default_rng(1).uniform(-1, 1, sys_.nDofs))
    sys_.setTime(0.0, 500.0)
    sys_.setToZero()
    sys_.assembleMatrices()
    ia, ja = sys_.pattern()
    A = sp.csr_matrix((sys_.getMatrix(), ja, ia))
    blocks = np.zeros(sys_.nInc, int) if rows == 0 else num.setup(rows).blocks()
    r = np.random.default_rng(4).uniform(-1, 1, sys_.nInc)
    z, ref = sys_.applyPreconditioner(r), _ilu_reference(A, r, blocks)
    assert np.max(np.abs(z - ref)) <= (1e-11 if precision == "fp64" else 1e-2) * np.max(np.abs(ref))


LATE = r"""
import json, sys
import numpy as np
import feng_gb300 as fe
sys.path.insert(0, "tests")
from helpers import problem_spaces
precision, rows, krylov = sys.argv[1], int(sys.argv[2]), sys.argv[3]
num, forms = problem_spaces("diffusion", fe.Mesh2DP1.generate_square(20, jitter=0.1, seed=2))
s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(
    krylov=krylov, precond="ilu0" if rows == 0 else "bjacobi-ilu0", pc_block_rows=max(rows, 1), precision=precision))
s.setToZero()
s.assembleResiduals()
s.assembleMatrices()
z = s.applyPreconditioner(np.random.default_rng(4).uniform(-1, 1, s.nInc))
st = s.solve(raise_on_failure=False)
print(json.dumps([int(np.isfinite(z).sum()), len(z), st["status"], bool(np.all(np.isfinite(s.getMatrix())))]))
"""


@pytest.mark.parametrize("krylov,precision,rows,step", [("fgmres", "fp64", 0, k) for k in (0, 1, 2, 3, 4, 5, 60)] +
                         [("fgmres", "mixed", 0, 7), ("fgmres", "fp64", 256, 0), ("fgmres", "fp64", 256, 6),
                          ("fgmres", "fp64", 0, 4095), ("cg", "fp64", 0, 1), ("cg", "fp64", 0, 4095)])
def test_a_late_copy_ends_the_solve_without_a_result(krylov, precision, rows, step):
    """Where a step's operands do not come in time (FENG_ILU_LATE_STEP: a step
    that counts as late) the whole of z is NaN, whatever lay in the stage, the
    solve says that it is not finite, and the GPU goes on working.  Steps
    among those asked for at the start, behind them and far behind them; one
    that does not exist changes nothing."""
    r = subprocess.run([sys.executable, "-c", LATE, precision, str(rows), krylov], cwd=ROOT,
                       env=dict(os.environ, FENG_ILU_LATE_STEP=str(step)), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    finite, n, status, matrix = json.loads(r.stdout.splitlines()[-1])
    assert n > 0 and matrix
    assert (finite, status) == ((n, 0) if step == 4095 else (0, -7))


def _block_entries(s, blocks):
    ia, ja = s.pattern()
    return int(np.sum(blocks[np.repeat(np.arange(s.nInc), np.diff(ia))] == blocks[ja]))


@pytest.mark.parametrize("rows", [8, 24, 256])
def test_block_jacobi_memory_stays_near_the_factor(rows):
    """A system of many diagonal blocks holds, beside the factor (FP64 value,
    column and position in the matrix: 16 bytes an entry), at most 4 values and
    1.1 column words (of 16 bytes) an entry packed for the solves, and 64 bytes a
    row of schedules.  A count of the packing on this mesh gives 3.2 and 3.7
    values and 1.0 column words an entry with blocks of 24 and 256 rows (blocks
    of 8 rows are not packed)."""
    torch = pytest.importorskip("torch")
    from feng_gb300 import kovasznay
    _, num, forms = kovasznay.build(128)
    blocks = num.setup(rows).blocks()
    used = {}
    for precond in ("none", "bjacobi-ilu0", "none", "bjacobi-ilu0"):
        before = torch.cuda.mem_get_info()[0]
        s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(precond=precond, pc_block_rows=rows))
        used[precond] = before - torch.cuda.mem_get_info()[0]
        entries = _block_entries(s, blocks)
        del s
    extra = used["bjacobi-ilu0"] - used["none"]
    assert 0 < extra <= (16 + 4 * 8 + 1.1 * 16) * entries + 64 * len(blocks)


@pytest.mark.parametrize("rows", [8, 24, 96])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_ilu0_solves_match_serial_over_block_sizes(precision, rows):
    """Blocks of few rows (by levels), of the fewest that are solved in shared
    memory (24 rows in FP64, 96 in FP32: a warp alone in most steps, stored
    with the lanes that it uses) and of more.  Tolerance as for the smaller
    diffusion systems above: rounding, no growth (1e-12 and 1e-5 of max |z|)."""
    import scipy.sparse as sp
    num, forms = problem_spaces("diffusion", fe.Mesh2DP1.generate_square(23, jitter=0.1, seed=2), 40.0)
    s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(
        krylov="fgmres", precond="bjacobi-ilu0", pc_block_rows=rows, precision=precision))
    s.setToZero()
    s.assembleMatrices()
    ia, ja = s.pattern()
    A = sp.csr_matrix((s.getMatrix(), ja, ia))
    r = np.random.default_rng(4).uniform(-1, 1, s.nInc)
    z, ref = s.applyPreconditioner(r), _ilu_reference(A, r, num.setup(rows).blocks())
    assert np.max(np.abs(z - ref)) <= (1e-12 if precision == "fp64" else 1e-5) * np.max(np.abs(ref))


@pytest.mark.parametrize("precision,n", [("fp64", 80), ("mixed", 120)])
def test_ilu0_block_above_shared_memory_matches_serial(precision, n):
    """One block of more rows than shared memory holds (25,281 in FP64, 57,121
    in FP32): solved by levels.  Tolerances of the 64 x 64 system."""
    num, forms = problem_spaces("diffusion", fe.Mesh2DP1.generate_square(n, jitter=0.1, seed=2))
    s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(krylov="fgmres", precond="ilu0",
                                                                         precision=precision))
    s.setToZero()
    s.assembleMatrices()
    st = num.setup()
    ia, ja = s.pattern()
    off, el = st.coloring()
    g = {"tri": num.mesh.arrays()["tri"], "adr": st.elementDofs(), "nInc": s.nInc, "nDofs": s.nDofs,
         "color_offsets": off, "color_elements": el, "ia": ia, "ja": ja, "quad_degree": 4}
    r = np.random.default_rng(3).uniform(-1, 1, s.nInc)
    z, ref = s.applyPreconditioner(r), _oracle_ilu(g, s.getMatrix(), r)
    assert np.max(np.abs(z - ref)) <= (1e-12 if precision == "fp64" else 1e-5) * np.max(np.abs(ref))
