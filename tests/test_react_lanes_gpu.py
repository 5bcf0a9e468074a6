"""The Air-11 source's four-lanes-per-node kernel at the edges of its layout: blocks that leave lanes,
warps and CTAs partly empty (8 nodes a warp, 32 a CTA), extra state columns, in place and out of place,
and iteration counts before and after the Newton iterations settle; against the oracle over all nodes.

Tolerance: 1e-10 of the node's density.  The mixtures are those whose Newton matrices are well
conditioned, so round-off (1e-16) grows by a few orders of magnitude at most."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(elements, nodes, extra, seed):
    rng = np.random.default_rng(seed)
    u = rng.random((elements, nodes, 10))
    es = 2.5 * np.exp(u[..., 0] * np.log(40.0))
    hot = np.clip((es - 25.0) / 50.0, 0.0, 1.0)
    rad = 1e-3 + 2e-2 * hot
    Y = np.zeros((elements, nodes, 11))
    ions = 1e-6 * (0.01 + hot) * u[..., 1]
    Y[..., 3], Y[..., 0] = 30.0055 * ions, 5.4858e-4 * ions
    Y[..., 6], Y[..., 7], Y[..., 8] = 0.3 * rad * u[..., 2], rad * u[..., 3], rad * u[..., 4]
    Y[..., 10] = 0.233 - Y[..., 7] - Y[..., 8] * 16.0 / 30.0
    Y[..., 9] = 1.0 - Y.sum(-1)
    rho = 0.5 + 6.0 * u[..., 5]
    vel = np.stack([9.0 * u[..., 6], u[..., 7] - 0.5, u[..., 8] - 0.5], -1)
    E = rho * (es + 0.5 * (vel * vel).sum(-1))
    return np.concatenate([rho[..., None], rho[..., None] * vel, E[..., None], rho[..., None] * Y,
                           rng.random((elements, nodes, extra))], -1)


@pytest.mark.parametrize("elements,nodes", [(1, 1), (1, 7), (3, 11), (1, 32), (5, 13)])
@pytest.mark.parametrize("iterations", [0, 1, 3, 12])
def test_partly_filled_warps(elements, nodes, iterations):
    import torch
    from jax_fluid_sim_b200 import ReactingFlowCoupler
    from oracle.chemistry import Coupler, batch_react_block
    kw = dict(dimensionless=True, reference_temperature=220.0, reference_pressure=500.0, reference_length=0.2,
              max_newton_iters=iterations)
    U = _state(elements, nodes, extra=iterations % 2, seed=elements * 100 + nodes)
    ref = batch_react_block(Coupler(**kw), U[..., :16], 5.0e-5)
    coupler = ReactingFlowCoupler(**kw)
    dev = torch.as_tensor(U, device="cuda")
    out = coupler.react_block(dev, 5.0e-5)
    assert np.array_equal(dev.cpu().numpy(), U)
    got = out.cpu().numpy()
    assert np.array_equal(got[..., :5], U[..., :5]) and np.array_equal(got[..., 16:], U[..., 16:])
    assert np.abs(got[..., :16] - ref).max(-1).max() <= 1e-10 * U[..., 0].min()
    coupler.react_block(dev, 5.0e-5, out=dev)
    assert torch.equal(dev, out)
