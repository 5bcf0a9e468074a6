"""The nodal range that the warps' certificate works on is exact: an element whose certificate holds by a margin
far below single precision keeps its state bit for bit under the positivity limiter.  (One that it does not clear
comes back as mean + 1 * (U - mean), which loses the last bits of values well below the mean: the nodal momenta
here run through zero.)

Margins: 1e-9 of the density, where the certificate's own arithmetic rounds at 1e-15 times the Lebesgue constant (up
to 3.4) and the energy (up to 100), and a range rounded to single precision moves its bounds by 6e-8.  Also states
beyond single precision's range."""

import numpy as np
import pytest

from .test_limiter_certificate import certificate, lebesgue_from_tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e45])
@pytest.mark.parametrize("degree", [1, 2, 3])
def test_barely_cleared_elements_keep_their_bits(degree, scale):
    import torch
    from jax_fluid_sim_b200 import (HybridCompressibleSolver, HybridEulerOperator, HybridMesh, HybridPositivityLimiter,
                                    meshgen)
    solver = HybridCompressibleSolver(HybridMesh(meshgen.box_hex((6, 5, 4), hi=(6.0, 5.0, 4.0))),
                                      polynomial_degree=degree)
    op = HybridEulerOperator(solver)
    lim = HybridPositivityLimiter(op)
    L = lebesgue_from_tables(op.plan)
    floors = (lim.density_floor, lim.pressure_floor, lim.relative_floor)
    bp = op.plan.blocks[0]
    rng = np.random.default_rng(degree)
    U = np.empty((bp.E, bp.Np, 5))
    for e in range(bp.E):
        u = np.ones((bp.Np, 5)) + 0.01 * rng.standard_normal((bp.Np, 5))
        u[:, 1:4] = 0.3 * rng.standard_normal((bp.Np, 3)) * 10.0 ** rng.uniform(-3, 0, (bp.Np, 3))
        u[:, 4] = 0.05 * rng.standard_normal(bp.Np)
        lo, hi = -10.0, 100.0                    # energies that the certificate refuses and clears
        for _ in range(100):
            mid = 0.5 * (lo + hi)
            lo, hi = (lo, mid) if certificate(scale * (u + mid * np.eye(5)[4]), L, *floors) else (mid, hi)
        u[:, 4] += hi + 1e-9
        U[e] = scale * u
        assert certificate(U[e], L, *floors)
    dev = torch.as_tensor(U, device="cuda")
    out = lim({op.names[0]: dev})[op.names[0]]
    assert torch.equal(out, dev)
