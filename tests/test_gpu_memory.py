"""Device memory of a system goes back with it: systems of each preconditioner
that are created, used and dropped in turn leave no more behind than the first
one did (the context's own pools), within the allocator's 2 MiB pages."""
import gc

import numpy as np
import pytest

import feng_gb300 as fe
from feng_gb300 import cavity, cube, kovasznay

pytestmark = pytest.mark.gpu


def _use(kind, precision, precond):
    build = {"steady": lambda: kovasznay.build(48), "step_2d": lambda: cavity.build(48, 400.0),
             "step_3d": lambda: cube.build(8, 100.0)}[kind]
    _, num, forms = build()
    s = fe.createLinearSystem(fe.CUDA, forms, num, fe.LinearSolverOptions(precond=precond, precision=precision))
    sol = fe.feSolution(s)
    sol.initializeEssentialBC()
    if kind != "steady":
        fe.createTimeIntegrator(fe.BDF2, fe.feNLSolverOptions(), s, sol, 0.0, 1.0, 100)
        s.setTime(0.0, 150.0)
    s.setSolution(sol.u)
    s.setToZero()
    s.assembleResiduals()
    s.assembleMatrices()
    s.applyPreconditioner(np.ones(s.nInc))


@pytest.mark.parametrize("kind,precond", [("steady", "amg"), ("step_2d", "amg"), ("step_3d", "amg"),
                                          ("steady", "ilu0"), ("steady", "bjacobi-ilu0"), ("steady", "none")])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_dropped_systems_leave_no_device_memory(kind, precond, precision):
    torch = pytest.importorskip("torch")
    free = []
    for _ in range(4):
        _use(kind, precision, precond)
        gc.collect()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - min(free[1:]) <= 2 << 20, free
