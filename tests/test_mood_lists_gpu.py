"""The MOOD step's certificate lists (k_blend_certify, k_hex_positivity; csrc/aux_kernels.cuh) from states where no
element misses its certificate to strong fronts, with element counts that leave the last CTA part full;
against the oracle's step."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("shape", [(3, 3, 3), (5, 3, 3)])
@pytest.mark.parametrize("jump", [0.01, 8.0, 4000.0])
def test_mood_step_against_oracle(jump, shape, degree):
    import jax_fluid_sim_b200 as jfs
    from jax_fluid_sim_b200 import meshgen
    from oracle.dg import Operator, PositivityLimiter, TimeIntegrator
    from oracle.mesh import Mesh, MeshSource
    from oracle.physics import FarfieldWallBoundary, Gas
    from oracle.subcell import MOODLimiter
    src = meshgen.box_hex(shape, hi=tuple(float(n) for n in shape), jitter=0.1, seed=3)
    solver = jfs.HybridCompressibleSolver(jfs.HybridMesh(src), polynomial_degree=degree)
    op = jfs.HybridEulerOperator(solver)
    om = Mesh(MeshSource(src.points, src.cells, src.physical, src.field_data, src.periodic_map))
    oop = Operator(om, Gas(), degree)
    far = [1.0, 0.3, 0.1, 0.0, 1.0]
    bc, obc = jfs.FarfieldWallBoundary(solver, far), FarfieldWallBoundary(oop.gas, om.physical_names, far)

    def primitive(x):        # a front across the middle, waves everywhere
        s = 0.5 + 0.5 * np.tanh(4.0 * (x[..., 0] - 0.4 * shape[0]))
        w = np.sin(2.0 * x[..., 1]) * np.cos(2.0 * x[..., 2])
        p = (1.0 + 0.05 * w) * (1.0 + jump * s) / (1.0 + jump)
        return np.stack([1.0 + 0.2 * s, 0.3 + 0.1 * w, 0.1 * w, 0.0 * w, p], -1)

    U = solver.state_blocks_from_primitive_function(op, primitive)
    Uh = {k: v.cpu().numpy() for k, v in U.items()}
    lim = jfs.HybridMOODSubcellLimiter(op, positivity=jfs.HybridPositivityLimiter(op))
    got, valid, _, _ = jfs.HybridSSPRK3(op, cfl=0.3, limiter=lim).checked_step(U, 2e-3, bc)
    olim = MOODLimiter(oop, positivity=PositivityLimiter(oop))
    want, ok, _, _ = TimeIntegrator(oop, cfl=0.3, limiter=olim).checked_step(Uh, 2e-3, obc)
    assert valid == ok
    for k in want:
        # the limiter's theta is a bisection of 30 steps: 1e-9 of the state per application, two per stage
        assert np.abs(got[k].cpu().numpy() - want[k]).max() <= 1e-8 * np.abs(want[k]).max()
