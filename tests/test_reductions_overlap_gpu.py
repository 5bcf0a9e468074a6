"""The stable time step on one stream while checked steps of the same plan run on another: the two reductions have
launches of different sizes and must share neither partials nor the counter that finds the last CTA, or a result,
and with a counter left off zero every later one, is formed from partials that are not all there.  Results are minima
and maxima, so they are equal bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3, 3), (14, 13, 12)])
def test_stable_dt_beside_steps(shape):
    import torch
    from jax_fluid_sim_b200 import HybridCompressibleSolver, HybridEulerOperator, HybridMesh, HybridSSPRK3, meshgen
    src = meshgen.hybrid_box(shape, hi=tuple(float(n) for n in shape), jitter=0.1, seed=4)
    solver = HybridCompressibleSolver(HybridMesh(src), polynomial_degree=2)
    op = HybridEulerOperator(solver)
    rng = np.random.default_rng(1)

    def primitive(x):
        s = 1.0 + 0.1 * rng.random(x.shape[:-1])
        return np.stack([s, 0.5 * s, 0.1 * s, -0.1 * s, 1.0 + 0.2 * s], -1)

    U = solver.state_blocks_from_primitive_function(op, primitive)
    rate, step = HybridSSPRK3(op), HybridSSPRK3(op)
    want_dt = rate.stable_dt(U)
    work = {k: v.clone() for k, v in U.items()}
    want = step.checked_step_inplace(work, 1e-6).clone()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(60):
        for k, v in U.items():
            work[k].copy_(v)
        status = step.checked_step_inplace(work, 1e-6)
        with torch.cuda.stream(side):
            dt = rate.stable_dt_device(U)
    torch.cuda.synchronize()
    assert float(dt.item()) == want_dt and torch.equal(status, want)
    assert rate.stable_dt(U) == want_dt
    assert rate.state_admissibility(U)[0]
