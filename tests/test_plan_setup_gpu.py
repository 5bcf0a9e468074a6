"""What a plan's set-up leaves to its first call: the tables that set-up kernels write on the default stream are
there for a first right-hand side on a stream that does not synchronise with it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mu", [0.0, 0.02])
@pytest.mark.parametrize("mesh", ["box_hex", "mixed_block"])
def test_first_call_on_another_stream(mesh, mu):
    import torch
    from jax_fluid_sim_b200 import (FarfieldWallBoundary, HybridCompressibleSolver, HybridEulerOperator, HybridMesh,
                                    HybridNavierStokesOperator, meshgen)
    src = meshgen.mixed_block(jitter=0.1, seed=2) if mesh == "mixed_block" else meshgen.box_hex(
        (12, 12, 12), hi=(12.0,) * 3, jitter=0.1, seed=3)
    solver = HybridCompressibleSolver(HybridMesh(src), polynomial_degree=2, dynamic_viscosity=mu)
    op = (HybridNavierStokesOperator if mu else HybridEulerOperator)(solver)
    bc = FarfieldWallBoundary(solver, [1.0, 0.4, 0.1, 0.0, 1.0])

    def primitive(x):
        s = 1.0 + 0.2 * np.sin(1.3 * x[..., 0]) * np.cos(0.7 * x[..., 1])
        return np.stack([s, 0.5 * s, 0.1 * np.sin(x[..., 2]), 0.0 * s, 1.0 + 0.5 * s], -1)

    U = solver.state_blocks_from_primitive_function(op, primitive)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        first = op.with_precision("float64").rhs(U, bc)
    torch.cuda.synchronize()
    again = op.rhs(U, bc)
    assert all(torch.equal(first[k], again[k]) for k in again)


@pytest.mark.parametrize("points", [8, 682, 683, 1200])
def test_volume_rules_of_any_size_are_accepted(points):
    """A block with more volume points than fit one CTA's default shared memory (683 of 9 values)."""
    import ctypes
    from jax_fluid_sim_b200 import _native as N
    L = N.lib()
    prm = N.Params()
    prm.degree, prm.nvars, prm.num_blocks, prm.gamma, prm.gas_constant = 1, 5, 1, 1.4, 1.0
    handle = ctypes.c_void_p()
    N.check(L.dgb_plan_create(ctypes.byref(prm), ctypes.byref(handle)))
    try:
        arrays = dict(basis=np.ones((points, 8)), basis_grad=np.ones((points, 8, 3)),
                      inv_jacobian=np.ones((2, points, 3, 3)), wdet=np.ones((2, points)), length=np.ones(2),
                      face_sample_basis=np.ones((4, 8)), p1_projector=np.eye(8), inv_mass=np.ones((2, 8, 8)))
        faces = np.arange(12, dtype=np.int32)
        d = N.BlockDesc(element_type=0, num_elements=2, num_nodes=8, num_qp=points, num_local_faces=6,
                        elem_face=N.dptr(faces, ctypes.c_int32), num_face_samples=4)
        for k, a in arrays.items():
            setattr(d, k, N.dptr(a))
        N.check(L.dgb_plan_set_block(handle, 0, ctypes.byref(d)))
    finally:
        L.dgb_plan_destroy(handle)


def test_split_residuals_are_the_only_outputs_allocated():
    """A plan that forms the residuals apart (the six-launch hexahedron form) allocates them and their sum, three
    states, and no output for the single residual that it does not have; switching the form back takes that one."""
    import torch
    from jax_fluid_sim_b200 import HybridCompressibleSolver, HybridMesh, HybridNavierStokesOperator, meshgen
    solver = HybridCompressibleSolver(HybridMesh(meshgen.box_hex((16, 16, 16), hi=(1.0,) * 3, jitter=0.1, seed=3)),
                                      polynomial_degree=2, dynamic_viscosity=0.02)
    op = HybridNavierStokesOperator(solver)
    U = solver.state_blocks_from_primitive_function(
        op, lambda x: np.stack([1.0 + 0.1 * np.sin(x[..., 0]), 0.3 + 0 * x[..., 0], 0 * x[..., 1], 0 * x[..., 2],
                                1.0 + 0 * x[..., 0]], -1))
    state = sum(v.numel() * 8 for v in U.values())
    for fused, states in ((True, 1), (False, 3), (True, 1)):
        op.native.set_fused(fused)
        op.rhs(U)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        R = op.rhs(U)
        assert torch.cuda.max_memory_allocated() - before < (states + 0.5) * state
        del R
