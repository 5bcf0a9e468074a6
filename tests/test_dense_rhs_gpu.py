"""The two-launch right-hand side of the dense path (csrc/dense_rhs.cu) where its CTAs are not
full: one element of each type, a few elements with boundary faces, and boxes whose element counts leave
remainders, at every degree; against the oracle's residual and checked step."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MESHES = {
    "one_of_each": lambda m: m.smoke_mesh(),
    "mixed_block": lambda m: m.mixed_block(jitter=0.1, seed=2),
    "box_3": lambda m: m.hybrid_box((3, 3, 3), hi=(3.0,) * 3, jitter=0.1, seed=4),
    "box_5": lambda m: m.hybrid_box((5, 3, 4), hi=(5.0, 3.0, 4.0), jitter=0.1, seed=5),
}


def _cases(mesh, degree, precision="float64", affine=True, mu=0.0):
    from jax_fluid_sim_b200 import (FarfieldWallBoundary, HybridCompressibleSolver, HybridEulerOperator, HybridMesh,
                                    HybridNavierStokesOperator, meshgen)
    from oracle.dg import Operator
    from oracle.mesh import Mesh, MeshSource
    from oracle.physics import FarfieldWallBoundary as OracleBoundary
    from oracle.physics import Gas
    src = MESHES[mesh](meshgen)
    solver = HybridCompressibleSolver(HybridMesh(src), polynomial_degree=degree, dynamic_viscosity=mu)
    op = (HybridNavierStokesOperator if mu else HybridEulerOperator)(solver, precision=precision, affine=affine)
    om = Mesh(MeshSource(src.points, src.cells, src.physical, src.field_data, src.periodic_map))
    oop = Operator(om, Gas(dynamic_viscosity=mu), degree)
    far = [1.0, 0.8, 0.1, -0.05, 1.0]
    bc = obc = None
    if src.periodic_map is None:
        bc, obc = FarfieldWallBoundary(solver, far), OracleBoundary(oop.gas, om.physical_names, far)

    def primitive(x):
        s = 1.0 + 0.1 * np.sin(2.0 * x[..., 0] + 0.3) * np.cos(1.5 * x[..., 1]) * np.cos(x[..., 2])
        return np.stack([s, 0.5 * s, 0.2 + 0.1 * np.sin(x[..., 2]), -0.1 * s, 1.0 + 0.2 * (s - 1.0)], -1)

    U = solver.state_blocks_from_primitive_function(op, primitive)
    return op, oop, bc, obc, U, {k: v.cpu().numpy() for k, v in U.items()}


@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_residual_and_step_against_oracle(mesh, degree):
    from jax_fluid_sim_b200 import HybridSSPRK3
    from oracle.dg import TimeIntegrator
    op, oop, bc, obc, U, Uh = _cases(mesh, degree)
    ref = oop.inviscid_rhs(Uh, obc)
    got = op.rhs(U, bc)
    for k in ref:
        assert np.abs(got[k].cpu().numpy() - ref[k]).max() <= 1e-9 * max(np.abs(r).max() for r in ref.values())
    stepped, valid, _, _ = HybridSSPRK3(op, cfl=0.3).checked_step(U, 1e-4, bc)
    want, ok, _, _ = TimeIntegrator(oop, cfl=0.3).checked_step(Uh, 1e-4, obc)
    assert valid == ok
    for k in want:
        assert np.abs(stepped[k].cpu().numpy() - want[k]).max() <= 1e-9 * np.abs(want[k]).max()


@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("affine", [True, False])
def test_mixed_precision_residual(degree, affine):
    op, oop, bc, obc, U, Uh = _cases("box_5", degree, "mixed", affine)
    ref = oop.inviscid_rhs(Uh, obc)
    got = op.rhs(U, bc)
    for k in ref:        # the bar of mixed residuals on hybrid boxes
        assert np.abs(got[k].cpu().numpy() - ref[k]).max() <= 5e-5 * max(np.abs(r).max() for r in ref.values())


@pytest.mark.parametrize("affine", [True, False])
@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_viscous_residual_and_step_against_oracle(mesh, degree, affine):
    """The whole residual as one, against the oracle's sum and against the separate right-hand sides."""
    from jax_fluid_sim_b200 import HybridSSPRK3
    from oracle.dg import TimeIntegrator
    op, oop, bc, obc, U, Uh = _cases(mesh, degree, affine=affine, mu=0.02)
    ref = oop.rhs(Uh, obc)
    got, inv, vis = op.rhs(U, bc), op.inviscid_rhs(U, bc), op.viscous_rhs(U, bc)
    scale = max(np.abs(r).max() for r in ref.values())
    for k in ref:
        assert np.abs(got[k].cpu().numpy() - ref[k]).max() <= 1e-9 * scale
        assert (got[k] - inv[k] - vis[k]).abs().max().item() <= 1e-9 * scale
    stepped, valid, _, _ = HybridSSPRK3(op, cfl=0.3).checked_step(U, 1e-4, bc)
    want, ok, _, _ = TimeIntegrator(oop, cfl=0.3).checked_step(Uh, 1e-4, obc)
    assert valid == ok
    for k in want:
        assert np.abs(stepped[k].cpu().numpy() - want[k]).max() <= 1e-9 * np.abs(want[k]).max()
