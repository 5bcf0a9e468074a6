"""dgb_subcell_recompute into the buffers of its own inputs: the result in a buffer of its own, in the
candidate's, in the base state's and in the additional right-hand side's is the same bit for bit (each element is
written last, from what has been read; the work lists' order enters no result), and the inputs that are not the output
keep their values.  From no troubled element to all of them, on a mesh of every element type and on hexahedra, fewer and
more than one wave of CTAs (out of place, large candidates are copied first)."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("mesh", ["mixed_block", "box_hex", "large_box_hex"])
def test_output_in_an_input_buffer(mesh, degree, share):
    import torch
    from jax_fluid_sim_b200 import (FarfieldWallBoundary, HybridCompressibleSolver, HybridMesh, HybridNavierStokesOperator,
                                    HybridSubcellFV, meshgen)
    from jax_fluid_sim_b200 import _native as N
    src = meshgen.mixed_block(jitter=0.1, seed=2) if mesh == "mixed_block" else meshgen.box_hex(
        (4, 3, 2) if mesh == "box_hex" else (12, 12, 12), hi=(4.0, 3.0, 2.0), jitter=0.1, seed=3)
    solver = HybridCompressibleSolver(HybridMesh(src), polynomial_degree=degree, dynamic_viscosity=0.02)
    op = HybridNavierStokesOperator(solver)
    fv = HybridSubcellFV(op)
    bc = FarfieldWallBoundary(solver, [1.0, 0.4, 0.1, 0.0, 1.0])

    def primitive(x, shift=0.0):
        s = 1.0 + 0.3 * np.tanh(4.0 * (x[..., 0] - 1.1 - shift)) * np.cos(x[..., 1])
        return np.stack([s, 0.5 * s, 0.1 * np.sin(x[..., 2]), 0.0 * s, 1.0 + 0.5 * s], -1)

    base = solver.state_blocks_from_primitive_function(op, primitive)
    cand = solver.state_blocks_from_primitive_function(op, lambda x: primitive(x, 0.2))
    arhs = {k: 0.05 * torch.cos(17.0 * v) for k, v in base.items()}
    g = torch.Generator().manual_seed(degree)
    flags = {k: (torch.rand(v.shape[0], generator=g) < share).to(torch.uint8).cuda() for k, v in base.items()}
    dt = 1e-3
    want = fv.recompute(base, cand, dt, flags, bc, arhs)
    if share == 0.0:
        assert all(torch.equal(want[k], cand[k]) for k in want)
    fp = (ctypes.c_void_p * N.MAX_BLOCKS)(*[flags[k].data_ptr() for k in op.names])
    for target in ("base", "cand", "arhs"):
        given = dict(base=base, cand=cand, arhs=arhs)
        bufs = {n: {k: v.clone() for k, v in s.items()} for n, s in given.items()}
        st = {n: op.native.state(op._blocks(s)) for n, s in bufs.items()}
        N.check(N.lib().dgb_subcell_recompute(op.native.handle, ctypes.byref(st["base"]), ctypes.byref(st["cand"]), dt,
                                              ctypes.byref(st["arhs"]), fp, ctypes.byref(st[target]),
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        for k in want:
            assert torch.equal(bufs[target][k], want[k]), (target, k)
            for n in bufs:
                assert n == target or torch.equal(bufs[n][k], given[n][k])
