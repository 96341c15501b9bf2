"""The scale pass of an Arnoldi step inside the next step's preconditioner
(replayed parts of a cycle) against the pass by itself (FENG_CUDA_GRAPHS=0,
where the host looks at the estimate after every step): the same basis to
rounding, so both solutions within the solves' 1e-10 of the matrix's, times a
factor of 100 for its condition on these meshes.

Restart lengths below, at and beside the parts' five steps; a few rows, and
more than one block of them."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SNIPPET = r"""
import json, sys
import numpy as np
from feng_gb300 import api as fe, kovasznay
out = []
for n, restart in json.loads(sys.argv[2]):
    _, num, forms = kovasznay.build(n)
    s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(
        precond="amg", precision=sys.argv[1], rel_tol=1e-10, restart=restart, max_iter=5000))
    sol = fe.feSolution(s)
    sol.initializeEssentialBC()
    s.setSolution(sol.u)
    s.setToZero()
    s.assembleResiduals()
    s.assembleMatrices()
    st = s.solve()
    out.append(s.getDu())
np.savez(sys.argv[3], *out)
"""
SIZES = [(3, 4), (12, 5), (24, 12), (24, 50)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pass_inside_and_alone_agree(precision, tmp_path):
    got = []
    for graphs in ("1", "0"):
        f = tmp_path / f"g{graphs}.npz"
        r = subprocess.run([sys.executable, "-c", SNIPPET, precision, json.dumps(SIZES), str(f)], cwd=ROOT,
                           env=dict(os.environ, FENG_CUDA_GRAPHS=graphs), capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        with np.load(f) as z:
            got.append([z[k] for k in z.files])
    for a, b in zip(*got):
        assert np.all(np.isfinite(a))
        assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)


COUNTS = SNIPPET.replace("out.append(s.getDu())", "out.append(st['nIter'])").replace(
    "np.savez(sys.argv[3], *out)", "print(json.dumps(out))")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pass_inside_and_alone_take_the_same_steps(precision):
    """A wrong basis vector, rotation or scaled right-hand side that restarts
    from the true residual repair costs steps: the counts agree to rounding
    (one step, and in mixed precision one per restart)."""
    got = []
    for graphs in ("1", "0"):
        r = subprocess.run([sys.executable, "-c", COUNTS, precision, json.dumps(SIZES)], cwd=ROOT,
                           env=dict(os.environ, FENG_CUDA_GRAPHS=graphs), capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(json.loads(r.stdout.splitlines()[-1]))
    for (n, restart), a, b in zip(SIZES, *got):
        assert min(a, b) > restart or min(a, b) > 5
        assert abs(a - b) <= (1 if precision == "fp64" else 1 + min(a, b) // restart), (n, restart, a, b)
