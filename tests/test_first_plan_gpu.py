"""The first plan of a process: kernels whose dynamic shared memory together with their static arrays passes 48 KB
need their limit raised by their own launch, not by that of an earlier, larger plan.  One process per plan: viscous
right-hand sides of 5 and 16 variables on a mesh of every element type, at the degrees on both sides of the limit."""

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import numpy as np, torch
from jax_fluid_sim_b200 import AIR11_SPECIES, HybridCompressibleSolver, HybridMesh, HybridNavierStokesOperator, meshgen
mesh = HybridMesh(meshgen.hybrid_box((6, 6, 6), hi=(6.0,) * 3, jitter=0.1, seed=0))
species = tuple(s.name for s in AIR11_SPECIES) if {species} else ()
solver = HybridCompressibleSolver(mesh, species_names=species, polynomial_degree={degree}, dynamic_viscosity=0.01)
op = HybridNavierStokesOperator(solver, precision="{precision}")
U = {{}}
for bp in op.plan.blocks:
    u = np.zeros((bp.E, bp.Np, solver.layout.number_of_variables))
    u[..., 0], u[..., 1], u[..., 4] = 1.0, 0.5, 2.5
    if species:
        u[..., -1] = 1.0
    U[bp.etype] = torch.as_tensor(u, device="cuda")
for out in (op.viscous_rhs(U), op.inviscid_rhs(U), op.rhs(U)):
    assert all(bool(torch.isfinite(v).all()) for v in out.values())
    # a uniform flow stays (float32 gradients of a constant do not vanish to 1e-9)
    assert "{precision}" == "mixed" or all(float(v.abs().max()) < 1e-9 for v in out.values())
"""


@pytest.mark.parametrize("precision", ["float64", "mixed"])
@pytest.mark.parametrize("species", [False, True])
@pytest.mark.parametrize("degree", [1, 2, 3])
def test_viscous_right_hand_sides(degree, species, precision):
    run = subprocess.run([sys.executable, "-c", PROGRAM.format(degree=degree, species=species, precision=precision)],
                         cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-2000:]
