"""Wall forces of inviscid operators on hybrid meshes, whose right-hand side takes two launches and keeps no face
traces unless they are asked for: the force must be that of the state given, at once and for a second state.

The fluid is at rest with p = p0 + G . x, so the conserved state is linear in x and its traces are exact: the force
is the sum of p n dA over the wall's face points.  Tolerances, of the sum of |p| dA (and of |p| |r| dA for moments):
float64 1e-12 (sums of some hundred terms of 1e-16); mixed 1e-6 (traces minus the anchor state in float32: a
few roundings of 6e-8 of differences no larger than the state)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["float64", "mixed"])
@pytest.mark.parametrize("degree", [1, 2, 3])
def test_linear_pressure_on_a_hybrid_block(degree, precision):
    from jax_fluid_sim_b200 import (FarfieldWallBoundary, HybridCompressibleSolver, HybridEulerOperator, HybridMesh,
                                    meshgen)
    from jax_fluid_sim_b200.aerodynamics import AerodynamicForceCalculator, face_points
    solver = HybridCompressibleSolver(HybridMesh(meshgen.mixed_block(jitter=0.1, seed=2)), polynomial_degree=degree)
    op = HybridEulerOperator(solver, precision=precision)
    assert sorted(op.names) == ["hexahedron", "tetra", "wedge"]
    bc = FarfieldWallBoundary(solver, [1.0, 0.0, 0.0, 0.0, 1.0])
    center = np.array([0.2, 0.3, 0.1])
    calc = AerodynamicForceCalculator(op, bc, wall_tag_names=("walls",), moment_center=center)
    points = face_points(op.plan)
    tol = 1e-12 if precision == "float64" else 1e-6
    for p0, G in ((2.0, np.array([0.3, -0.2, 0.1])), (1.5, np.array([-0.1, 0.25, 0.2]))):
        def primitive(x):
            W = np.zeros(x.shape[:-1] + (5,))
            W[..., 0] = 1.0
            W[..., 4] = p0 + x @ G
            return W

        F, M, Fs, Ms = np.zeros(3), np.zeros(3), 0.0, 0.0
        for ftype, fp in op.plan.faces.items():
            wall = (fp.nbr_block < 0) & np.isin(fp.tags, calc.wall_tags)
            x, w = points[ftype][wall], fp.weights[wall]
            f = ((p0 + x @ G) * w)[..., None] * fp.normals[wall]
            F += f.sum((0, 1))
            M += np.cross(x - center, f).sum((0, 1))
            size = np.abs((p0 + x @ G) * w)
            Fs += size.sum()
            Ms += (size * np.linalg.norm(x - center, axis=-1)).sum()
        assert Fs > 1.0
        got = calc.forces_device(solver.state_blocks_from_primitive_function(op, primitive)).cpu().numpy()
        assert np.abs(got[0:3] - F).max() <= tol * Fs
        assert np.abs(got[3:6] - M).max() <= tol * Ms
        assert np.abs(got[6:]).max() == 0.0
