"""The work that a user of this framework has it do, as cases that can be timed and checked.

A case is a dict of plain values: ``family`` names the kind of call, the other entries its sizes
and options.  The families follow the framework's own configurations (``workloads.py``, ``bench.py``):

* ``rhs``        one right-hand side of the Navier-Stokes operator on a hybrid box, as a caller with
                 its own time integrator takes it;
* ``taylor``     the Taylor-Green loop: the stable dt of the state, read by the host, then one checked
                 step at it;
* ``vortex``     one checked Euler step of the isentropic vortex on hexahedra, prisms and tetrahedra,
                 replayed as a CUDA graph;
* ``cylinders``  one checked step of an ensemble of extruded cylinder grids joined into one plan;
* ``sphere``     one checked step of the Mach-3 viscous sphere (the headline configuration);
* ``reacting``   one checked step of the Mach-8 sphere with the 11 Air-11 species, then the source on
                 every node (the reacting driver's step);
* ``source``     the Air-11 source alone on a block of hot nodes.

Every stepped pass copies the state to advance into the buffers that the step works on, as a program
does that steps states which arrive from elsewhere.  ``exact`` evaluates the same discretisation with
plain torch in 64 bits: its own reference elements, quadrature, face pairing, metrics, fluxes,
lifting, limiter and chemistry.  It gives no value for a step with the MOOD subcell limiter: what that
leaves in a troubled element follows from the subcell scheme's index conventions, not from the
equations.
"""

import math

import numpy as np
import torch

from jax_fluid_sim_b200 import (FarfieldWallBoundary, HybridCompressibleSolver, HybridMesh,
                                HybridMOODSubcellLimiter, HybridNavierStokesOperator, HybridPositivityLimiter,
                                HybridSSPRK3, ReactingFlowCoupler, meshgen)
from jax_fluid_sim_b200 import workloads as wl
from jax_fluid_sim_b200.air11 import AIR11_REACTIONS, AIR11_SPECIES
from jax_fluid_sim_b200.ensemble import HybridEnsemble
from jax_fluid_sim_b200.operators import HybridEulerOperator

GAMMA = 1.4


# ------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # a handful of elements of every type: launches and latency; an external integrator's call
        dict(name="rhs_hybrid_4", family="rhs", n=4, degree=2, precision="float64"),
        # the Taylor-Green configuration at its own size, as its loop runs it
        dict(name="taylor_16_p2", family="taylor", n=16, degree=2, precision="float64"),
        # the order study's boxes: each degree, both precisions, small and large
        dict(name="vortex_16_p3", family="vortex", n=16, degree=3, precision="float64", tensor_cores=False),
        dict(name="vortex_32_p1", family="vortex", n=32, degree=1, precision="float64", tensor_cores=False),
        dict(name="vortex_23_p2_mixed", family="vortex", n=23, degree=2, precision="mixed", tensor_cores=False),
        # cylinder ensembles: uneven cases in one plan, and one case alone
        dict(name="cylinders_8_p2_mixed", family="cylinders", cases=8, smallest=500, largest=6000, degree=2,
             precision="mixed", limiter="positivity"),
        dict(name="cylinder_1_p3", family="cylinders", cases=1, smallest=3001, largest=3001, degree=3,
             precision="float64", limiter="positivity"),
        # the Mach-3 sphere: plain float64 on the medium grid, the headline (mixed, MOOD, full grid)
        dict(name="sphere_39k_p3", family="sphere", n=16, n_radial=10, up=4, down=16, side=6, degree=3,
             precision="float64", limiter="positivity"),
        dict(name="sphere_13k_p2_mood", family="sphere", n=11, n_radial=7, up=3, down=11, side=4, degree=2,
             precision="float64", limiter="mood"),
        dict(name="sphere_202k_p3_mixed_mood", family="sphere", n=24, n_radial=20, up=8, down=32, side=12, degree=3,
             precision="mixed", limiter="mood"),
        # the reacting sphere's step, and its source alone
        dict(name="reacting_7k_p2_mood", family="reacting", n=8, n_radial=6, up=3, down=10, side=4, degree=2,
             precision="float64"),
        dict(name="source_54k_nodes", family="source", elements=2000, nodes=27, iterations=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["rhs", "taylor", "vortex", "vortex", "cylinders", "cylinders", "sphere", "sphere", "sphere",
                         "reacting", "source"])
    degree = rng.choice([1, 2, 3])
    precision = rng.choice(["float64", "mixed"])
    if family == "rhs":
        return dict(family=family, n=rng.randint(3, 12), degree=degree, precision="float64")
    if family == "taylor":
        return dict(family=family, n=rng.randint(4, 32), degree=degree, precision=precision)
    if family == "vortex":
        return dict(family=family, n=_log_int(rng, 4, 32), degree=degree, precision=precision,
                    tensor_cores=precision == "mixed" and rng.random() < 0.5)
    if family == "cylinders":
        cases = rng.choice([1, 1, rng.randint(2, 16)])
        largest = _log_int(rng, 400, 6000)
        return dict(family=family, cases=cases, smallest=largest if cases == 1 else max(200, largest // 10),
                    largest=largest, degree=rng.choice([2, 3]), precision=precision,
                    limiter=rng.choice(["positivity", "mood"]))
    if family == "source":
        return dict(family=family, elements=_log_int(rng, 100, 8000), nodes=rng.choice([8, 27, 64]),
                    iterations=rng.choice([4, 12, 12]))
    n = rng.randint(4, 18 if family == "sphere" else 8)
    grid = dict(n=n, n_radial=max(2, round(n * rng.uniform(0.5, 0.9))), up=max(1, round(n * rng.uniform(0.2, 0.4))),
                down=max(3, round(n * rng.uniform(0.8, 1.3))), side=max(1, round(n * rng.uniform(0.3, 0.5))))
    if family == "reacting":
        return dict(family=family, **grid, degree=rng.choice([1, 2]), precision=precision)
    return dict(family=family, **grid, degree=degree, precision=precision, limiter=rng.choice(["mood", "positivity"]))


# ---------------------------------------------------------------------------------- meshes and set-up
def _sphere_source(case):
    return meshgen.sphere_oh_grid(n=case["n"], n_radial=case["n_radial"],
                                  outer=((case["up"], case["down"]),) + ((case["side"], case["side"]),) * 2)


def _sphere_elements(case):
    n, s = case["n"], 2 * case["side"]
    return (n + case["up"] + case["down"]) * (n + s) ** 2 - n ** 3 + 6 * n ** 2 * case["n_radial"]


def _ensemble(case):
    """(source, far-field primitive, viscosity) of every cylinder of the ensemble."""
    cases = wl.ensemble_cases(case["cases"], (case["smallest"], case["largest"]), seed=5, degrees=(case["degree"],))
    out = []
    for c in cases:
        far = np.array([1.0, c["mach"] * math.sqrt(GAMMA), 0.0, 0.0, 1.0])
        out.append((meshgen.cylinder_o_grid(c["n_theta"], c["n_radial"]), far, far[1] / c["reynolds"]))
    return out


def _waves(xyz, seed, channels, length=None):
    """Smooth random fields of unit size at the points xyz (..., 3): (..., channels); periodic in a
    box of side ``length`` if one is given."""
    g = torch.Generator().manual_seed(int(seed))
    out = torch.zeros(xyz.shape[:-1] + (channels,), dtype=torch.float64, device=xyz.device)
    for c in range(channels):
        for _ in range(3):
            if length is None:
                k = 3.0 * torch.rand(3, generator=g, dtype=torch.float64) - 1.5
            else:
                k = (2.0 * math.pi / length) * torch.randint(-2, 3, (3,), generator=g).double()
            phase = 2.0 * math.pi * torch.rand((), generator=g, dtype=torch.float64)
            out[..., c] += torch.sin(xyz @ k.to(xyz.device) + phase.item()) / 3.0
    return out


def _perturbed(W, xyz, seed, length=None, size=0.01):
    """Primitive states W with density and pressure changed by up to ``size`` and the velocity by
    up to ``size`` of the sound speed: the flow that the state has developed."""
    w = _waves(xyz, seed, 5, length)
    W = W.clone()
    c = torch.sqrt(GAMMA * W[..., 4] / W[..., 0])
    W[..., 0] *= 1.0 + size * w[..., 0]
    W[..., 4] *= 1.0 + size * w[..., 4]
    W[..., 1:4] += size * c[..., None] * w[..., 1:4]
    return W


def _conserved(W):
    rho, vel = W[..., :1], W[..., 1:4]
    E = W[..., 4:5] / (GAMMA - 1.0) + 0.5 * rho * (vel * vel).sum(-1, keepdim=True)
    return torch.cat([rho, rho * vel, E, rho * W[..., 5:]], -1)


def _shocked(xyz, far, radius=0.65):
    """The normal-shock state of the far field ``far`` in the elements whose nodes' mean lies inside
    r < radius, the far field elsewhere (the sphere configurations' start)."""
    far = torch.as_tensor(far, dtype=torch.float64, device=xyz.device)
    m2 = float(far[1] ** 2 / GAMMA)
    rho2 = (GAMMA + 1) * m2 / ((GAMMA - 1) * m2 + 2)
    inside = far.clone()
    inside[0], inside[1], inside[4] = rho2, far[1] / rho2, 1 + 2 * GAMMA / (GAMMA + 1) * (m2 - 1)
    near = (xyz.mean(dim=1).norm(dim=-1) < radius)[:, None, None]
    return torch.where(near, inside, far).expand(xyz.shape[:2] + far.shape)


def _primitive(case, etype, xyz, seed, case_id=None):
    """The primitive start at the solution nodes xyz (E, N, 3)."""
    family = case["family"]
    if family in ("vortex", "rhs"):
        W = torch.as_tensor(wl.vortex_primitive(xyz.cpu().numpy(), length=10.0), device=xyz.device)
        return _perturbed(W, xyz, seed, 10.0)
    if family == "taylor":
        W = torch.as_tensor(wl.tgv_primitive(xyz.cpu().numpy()), device=xyz.device)
        return _perturbed(W, xyz, seed, 2 * math.pi, 0.002)
    if family == "cylinders":
        far = torch.as_tensor(np.stack([e[1] for e in _ensemble(case)]), device=xyz.device)
        return _perturbed(far[case_id][:, None, :].expand(xyz.shape[:2] + (5,)), xyz, seed)
    if family == "sphere":
        far = np.array([1.0, wl.SPHERE_MACH * math.sqrt(GAMMA), 0.0, 0.0, 1.0])
        return _perturbed(_shocked(xyz, far), xyz, seed)
    return _perturbed(_shocked(xyz, wl.reacting_farfield()), xyz, seed)


def _start(case, op, seed, case_id=None):
    out = {}
    for name, xyz in op.solution_node_coordinates.items():
        xyz = torch.as_tensor(xyz, device="cuda")
        out[name] = _conserved(_primitive(case, name, xyz, seed, case_id)).contiguous()
    return out


def _flow(case):
    """(source or None, solver, operator, boundary, ensemble's case ids) of a flow case."""
    family, P = case["family"], case["degree"]
    if family == "cylinders":
        parts = _ensemble(case)
        ens = HybridEnsemble([p[0] for p in parts], [p[1] for p in parts], [p[2] for p in parts],
                             polynomial_degree=P, precision=case["precision"])
        ids = torch.cat([torch.full((len(p[0].cells[0][1]),), k) for k, p in enumerate(parts)]).cuda()
        return ens, ens.operator, ens.boundary, ids
    if family in ("vortex", "rhs"):
        src = meshgen.hybrid_box((case["n"],) * 3, hi=(10.0,) * 3, jitter=0.1, seed=0)
        mu, bc = (0.0 if family == "vortex" else 1e-2), None
    elif family == "taylor":
        src, mu, bc = wl.tgv_mesh(case["n"]), 1.0 / 1600.0, None
    else:
        src = _sphere_source(case)
        far = (wl.reacting_farfield() if family == "reacting"
               else np.array([1.0, wl.SPHERE_MACH * math.sqrt(GAMMA), 0.0, 0.0, 1.0]))
        mu = far[1] / (2.6e5 if family == "reacting" else wl.SPHERE_RE)
    species = tuple(s.name for s in AIR11_SPECIES) if family == "reacting" else ()
    solver = HybridCompressibleSolver(HybridMesh(src), species_names=species, gamma=GAMMA, polynomial_degree=P,
                                      dynamic_viscosity=mu, prandtl=0.71 if family == "taylor" else 0.72)
    kind = HybridEulerOperator if family == "vortex" else HybridNavierStokesOperator
    op = kind(solver, precision=case["precision"])
    if family in ("sphere", "reacting"):
        bc = FarfieldWallBoundary(solver, far, wall_temperature=wl.SPHERE_T_WALL / wl.SPHERE_T_INF)
    return solver, op, bc, None


def _coupler(iterations=12):
    return ReactingFlowCoupler(dimensionless=True, reference_temperature=wl.REACTING_T_INF,
                               reference_pressure=wl.REACTING_P_INF, reference_length=0.2, gamma=GAMMA,
                               max_newton_iters=iterations)


def _hot_nodes(case, seed):
    """Nodes of a Mach-8 flow: air from the free stream's thermal energy to three times that of a
    normal shock's, with traces of dissociated and ionised air in the cold part and percents of it in
    the hot part (mixtures whose Newton iterations converge, so that their result is defined)."""
    g = torch.Generator().manual_seed(int(seed))
    E, N = case["elements"], case["nodes"]
    u = torch.rand((E, N, 10), generator=g, dtype=torch.float64).cuda()
    es = 2.5 * torch.exp(u[..., 0] * math.log(40.0))                    # 2.5 to 100 (units of R T_ref)
    hot = ((es - 25.0) / 50.0).clamp(0.0, 1.0)
    radical = 1e-3 + 2e-2 * hot
    Y = torch.zeros((E, N, 11), dtype=torch.float64, device="cuda")
    # order: e-, N+, O+, NO+, N2+, O2+, N, O, NO, N2, O2
    ions = 1e-6 * (0.01 + hot) * u[..., 1]                              # NO+ with its electrons
    Y[..., 3], Y[..., 0] = 30.0055 * ions, 5.4858e-4 * ions
    Y[..., 6], Y[..., 7], Y[..., 8] = 0.3 * radical * u[..., 2], radical * u[..., 3], radical * u[..., 4]
    Y[..., 10] = 0.233 - Y[..., 7] - Y[..., 8] * (16.0 / 30.0)
    Y[..., 9] = 1.0 - Y.sum(-1)
    rho = 0.5 + 6.0 * u[..., 5]
    vel = torch.stack([9.0 * u[..., 6], u[..., 7] - 0.5, u[..., 8] - 0.5], -1)
    E_tot = rho * (es + 0.5 * (vel * vel).sum(-1))
    return torch.cat([rho[..., None], rho[..., None] * vel, E_tot[..., None], rho[..., None] * Y], -1).contiguous()


SOURCE_DT = 5.0e-5


def prepare(case, seed):
    family = case["family"]
    if family == "source":
        U = _hot_nodes(case, seed)
        return dict(case=case, U=U, out=torch.empty_like(U), coupler=_coupler(case["iterations"]))
    owner, op, bc, ids = _flow(case)
    U = _start(case, op, seed, ids)
    state = dict(case=case, owner=owner, op=op, bc=bc, U=U)
    if family == "rhs":
        return state
    limiter = None
    if case.get("limiter") or family == "reacting":
        limiter = HybridPositivityLimiter(op)
        if case.get("limiter", "mood") == "mood":
            limiter = HybridMOODSubcellLimiter(op, positivity=limiter)
    if case.get("tensor_cores"):
        op.native.set_tensor_cores(True)
    integ = HybridSSPRK3(op, cfl=0.3, limiter=limiter, graph=family != "taylor")
    state.update(integ=integ, work={k: torch.empty_like(v) for k, v in U.items()})
    if family != "taylor":
        state["dt"] = integ.stable_dt(U, bc)
    if family == "reacting":
        state["coupler"] = _coupler()
    return state


def run(state):
    case = state["case"]
    if case["family"] == "source":
        return state["coupler"].react_block(state["U"], SOURCE_DT, out=state["out"])
    if case["family"] == "rhs":
        return state["op"].rhs(state["U"], state["bc"])
    integ, work, bc = state["integ"], state["work"], state["bc"]
    for k, v in state["U"].items():
        work[k].copy_(v)
    dt = state["dt"] if "dt" in state else float(integ.stable_dt_device(work).item())
    status = integ.checked_step_inplace(work, dt, bc)
    out = dict(work)
    if case["family"] == "reacting":
        for k in work:
            state["coupler"].react_block(work[k], dt, out=work[k])
    out["valid"], out["minima"] = status.view(torch.int32)[:1], status[1:]     # admissible; least density, pressure
    return out


# -------------------------------------------------------------------------------- what a pass costs
def _points(etype, P):
    """(nodes, volume points, face points of one element) of the discretisation."""
    q = {1: 2, 2: 3, 3: 5}[P]
    quad, tri = {1: 4, 2: 9, 3: 16}[P], {1: 3, 2: 16, 3: 25}[P]
    if etype == "hexahedron":
        return (P + 1) ** 3, q ** 3, 6 * quad
    simplex = 125 if P > 1 else 4
    if etype == "wedge":
        return (P + 1) * (P + 1) * (P + 2) // 2, 125 if P > 1 else 6, 3 * quad + 2 * tri
    return (P + 1) * (P + 2) * (P + 3) // 6, simplex, 4 * tri


def _elements(case):
    family = case["family"]
    if family in ("vortex", "rhs"):
        cubes = case["n"] ** 3
        return {"hexahedron": 0.3 * cubes, "wedge": 0.88 * cubes, "tetra": 1.6 * cubes}
    if family == "taylor":
        return {"hexahedron": case["n"] ** 3}
    if family == "cylinders":
        cases = wl.ensemble_cases(case["cases"], (case["smallest"], case["largest"]), seed=5,
                                  degrees=(case["degree"],))
        return {"hexahedron": sum(c["n_theta"] * c["n_radial"] for c in cases)}
    return {"hexahedron": _sphere_elements(case)}


def _source_work(nodes, nvars, iterations):
    # per iteration: 22 reactions with two exponentials each (about 40 operations), 11 Gibbs energies,
    # their derivatives (about 900 products), an 11 x 11 elimination and three energy inversions
    per = 22 * 2 * 40 + 11 * 30 + 2 * 900 + 2 * 11 ** 3 / 3 + 3 * 11 * 20
    return 16.0 * nodes * nvars, nodes * iterations * per


def work(case):
    """The state in and out once, the mesh (corner points and connectivity) once; the products of the
    sum-factorised hexahedron and the dense prism and tetrahedron contractions, the fluxes, and the
    mass matrices, three times for a step."""
    if case["family"] == "source":
        nbytes, flops = _source_work(case["elements"] * case["nodes"], 16, case["iterations"])
        return {"bytes": nbytes, "flops": flops}
    P, nv = case["degree"], 16 if case["family"] == "reacting" else 5
    viscous = case["family"] != "vortex"
    nbytes = flops = nodes = 0.0
    for etype, count in _elements(case).items():
        Np, Nq, Nf = _points(etype, P)
        nodes += count * Np
        nbytes += count * (16.0 * Np * nv + 8 * 24 + 6 * 8)
        if etype == "hexahedron":
            n, q = P + 1, round(Nq ** (1 / 3))
            one = 2 * (n ** 3 * q + n ** 2 * q ** 2 + n * q ** 3)
            face = 2 * 6 * (n ** 3 + n ** 2 * q + n * q ** 2)
            per = one * nv * 4 + face * nv * 2 + 6 * n ** 4 * nv
            per += (one * (4 * 3 + 12) + face * (16 + 12)) if viscous else 0
        else:
            per = 2 * Nq * Np * nv * 4 + 2 * Nf * Np * nv * 2 + 2 * Np * Np * nv
            per += (2 * Nq * Np * (4 * 3 + 12) + 2 * Nf * Np * (16 + 12)) if viscous else 0
        per += Nq * (60 + 10 * nv + (80 if viscous else 0)) + Nf * (100 + 10 * nv + (80 if viscous else 0))
        flops += count * per * (1 if case["family"] == "rhs" else 3)
    if case["family"] == "reacting":
        b, f = _source_work(nodes, nv, 12)
        flops += f
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------- the same numbers in plain torch
_FACES = {
    "tetra": ((0, 2, 1), (0, 1, 3), (1, 2, 3), (2, 0, 3)),
    "wedge": ((0, 2, 1), (3, 4, 5), (0, 1, 4, 3), (1, 2, 5, 4), (2, 0, 3, 5)),
    "hexahedron": ((0, 3, 2, 1), (4, 5, 6, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7)),
}
_CORNERS = {
    "tetra": [[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]],
    "wedge": [[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [0, 1, 1]],
    "hexahedron": [[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]],
}
_LINE = {1: (0.0, 1.0), 2: (0.0, 1.0, 0.5), 3: (0.0, 1.0, 1.0 / 3.0, 2.0 / 3.0)}


def _t(x):
    return torch.as_tensor(np.asarray(x, dtype=np.float64), device="cuda")


def _nodes(etype, P):
    """Solution nodes in the state's order."""
    if P == 1:
        return _t(_CORNERS[etype])
    a, b = 1.0 / 3.0, 2.0 / 3.0
    if P == 2:
        tri = [(0, 0), (1, 0), (0, 1), (.5, 0), (.5, .5), (0, .5)]
        edges = [(.5, 0, 0), (0, .5, 0), (0, 0, .5), (.5, .5, 0), (.5, 0, .5), (0, .5, .5)]
    else:
        tri = [(0, 0), (1, 0), (0, 1), (a, 0), (b, 0), (b, a), (a, b), (0, b), (0, a), (a, a)]
        edges = [(a, 0, 0), (b, 0, 0), (0, a, 0), (0, b, 0), (0, 0, a), (0, 0, b), (b, a, 0), (a, b, 0), (b, 0, a),
                 (a, 0, b), (0, b, a), (0, a, b), (a, a, 0), (a, 0, a), (0, a, a), (a, a, a)]
    if etype == "tetra":
        return _t(_CORNERS["tetra"] + [list(e) for e in edges])
    if etype == "wedge":
        return _t([[x, y, z] for z in _LINE[P] for x, y in tri])
    return _t([[x, y, z] for z in _LINE[P] for y in _LINE[P] for x in _LINE[P]])


def _monomials(etype, P):
    """Exponents of the polynomial space that the nodes are unisolvent for."""
    r = range(P + 1)
    if etype == "hexahedron":
        return [(i, j, k) for k in r for j in r for i in r]
    if etype == "wedge":
        return [(i, j, k) for k in r for j in r for i in r if i + j <= P]
    return [(i, j, k) for k in r for j in r for i in r if i + j + k <= P]


def _basis(etype, P, pts):
    """Values (..., n) and gradients (..., n, 3) of the nodal basis at reference points."""
    ex = _monomials(etype, P)

    def powers(x):
        return torch.stack([x ** i for i in range(P + 1)], -1)

    def derivatives(x):
        return torch.stack([i * x ** max(i - 1, 0) for i in range(P + 1)], -1)

    def table(p):
        v = [powers(p[..., d]) for d in range(3)]
        g = [derivatives(p[..., d]) for d in range(3)]
        i, j, k = (torch.tensor(c, device="cuda") for c in zip(*ex))
        X, Y, Z = v[0][..., i], v[1][..., j], v[2][..., k]
        return X * Y * Z, torch.stack([g[0][..., i] * Y * Z, X * g[1][..., j] * Z, X * Y * g[2][..., k]], -1)

    inv = torch.linalg.inv(table(_nodes(etype, P))[0])                 # node values -> coefficients
    V, G = table(pts)
    return V @ inv, torch.einsum("...md,mn->...nd", G, inv)


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return list(zip(0.5 * (x + 1.0), 0.5 * w))


def _volume_rule(etype, P):
    if P == 1 and etype == "tetra":
        a, b = 0.5854101966249685, 0.1381966011250105
        return _t([[b, b, b], [a, b, b], [b, a, b], [b, b, a]]), _t([1.0 / 24.0] * 4)
    if P == 1 and etype == "wedge":
        rule = [((x, y, z), wz / 6.0) for z, wz in _gauss(2) for x, y in ((1 / 6, 1 / 6), (2 / 3, 1 / 6), (1 / 6, 2 / 3))]
    elif etype == "hexahedron":
        g = _gauss({1: 2, 2: 3, 3: 5}[P])
        rule = [((x, y, z), a * b * c) for z, a in g for y, b in g for x, c in g]
    elif etype == "wedge":
        g = _gauss(5)
        rule = [((a, (1 - a) * b, z), wa * wb * wz * (1 - a)) for z, wz in g for a, wa in g for b, wb in g]
    else:
        g = _gauss(5)
        rule = [((a, (1 - a) * b, (1 - a) * (1 - b) * c), wa * wb * wc * (1 - a) ** 2 * (1 - b))
                for a, wa in g for b, wb in g for c, wc in g]
    return _t([p for p, _ in rule]), _t([w for _, w in rule])


def _face_rule(corners, P):
    """Corner shapes (points, corners) and weights (measure of the reference face included)."""
    if corners == 3:
        if P == 1:
            return _t([[2 / 3, 1 / 6, 1 / 6], [1 / 6, 2 / 3, 1 / 6], [1 / 6, 1 / 6, 2 / 3]]), _t([1 / 6] * 3)
        g = _gauss(4 if P == 2 else 5)
        rule = [((1 - a - (1 - a) * b, a, (1 - a) * b), wa * wb * (1 - a)) for a, wa in g for b, wb in g]
    else:
        g = _gauss(P + 1)
        rule = [(((1 - u) * (1 - v), u * (1 - v), u * v, (1 - u) * v), wu * wv) for v, wv in g for u, wu in g]
    return _t([s for s, _ in rule]), _t([w for _, w in rule])


class _Plain:
    """The discretisation on one mesh: anchored Euler residual, HLLC, BR2, positivity limiter, SSP-RK3."""

    def __init__(self, src, P, prandtl=0.72, mu=0.0, far=None, wall_T=None, case_id=None):
        self.P, self.far, self.wall_T = P, far, wall_T
        self.br2 = (P + 1) * (P + 2) / 2
        pts = _t(src.points)
        canon = np.arange(len(src.points)) if src.periodic_map is None else np.asarray(src.periodic_map)
        canon = torch.as_tensor(canon, device="cuda").long()
        tags = {name: v[0] for name, v in src.field_data.items()}
        roles = dict(inlet=("inlet",), wall=("walls", "sphere_wall", "cylinder_wall", "symmetry"),
                     no_slip=("sphere_wall", "cylinder_wall"), slip=("walls", "symmetry"))
        self.roles = {r: [tags[n] for n in names if n in tags] for r, names in roles.items()}
        conn = {}
        for t in ("hexahedron", "wedge", "tetra"):
            parts = [np.asarray(c) for k, c in src.cells if k == t]
            if parts:
                conn[t] = torch.as_tensor(np.concatenate(parts), device="cuda").long()
        self.types, self.conn, self.xyz = list(conn), conn, {t: pts[c] for t, c in conn.items()}
        dev = dict(dtype=torch.float64, device="cuda")
        self.mu, self.kappa = {}, {}
        for t, c in conn.items():
            m = torch.as_tensor(mu, **dev)
            self.mu[t] = m[case_id] if case_id is not None else m.expand(len(c)).clone()
            self.kappa[t] = self.mu[t] * (GAMMA / (GAMMA - 1.0)) / prandtl
        self.viscous = bool(max(float(m.max()) for m in self.mu.values()) > 0)
        self.case_id = case_id
        self.B, self.wdet, self.grad, self.minv = {}, {}, {}, {}
        for t in self.types:
            q, w = _volume_rule(t, P)
            B, dB = _basis(t, P, q)
            J = torch.einsum("eid,qir->eqdr", self.xyz[t], _basis(t, 1, q)[1])
            self.B[t], self.wdet[t] = B, w * torch.linalg.det(J).abs()
            self.grad[t] = torch.einsum("qir,eqrd->eqid", dB, torch.linalg.inv(J))
            mass = torch.einsum("eq,qi,qj->eij", self.wdet[t], B, B)
            vol = self.wdet[t].sum(1)
            self.minv[t] = torch.clamp(vol / 1e-4, max=1.0)[:, None, None] * torch.linalg.inv(mass)
        self._faces(src, canon)

    def _faces(self, src, canon):
        """Faces by sorted corner ids: the first visit in block, element, local-face order owns."""
        key, blk, elem, loc, ids = [], [], [], [], []
        for b, t in enumerate(self.types):
            for c in (3, 4):
                which = [f for f, v in enumerate(_FACES[t]) if len(v) == c]
                if not which:
                    continue
                nodes = canon[self.conn[t][:, torch.tensor([_FACES[t][f] for f in which], device="cuda")]]   # E, f, c
                E = len(nodes)
                s = nodes.reshape(-1, c).sort(-1)[0]
                key.append((s[:, 0] << 42) | (s[:, 1] << 21) | s[:, 2])
                blk.append(torch.full((len(s),), b, device="cuda"))
                elem.append(torch.arange(E, device="cuda").repeat_interleave(len(which)))
                loc.append(torch.tensor(which, device="cuda").repeat(E))
                ids.append(torch.cat([nodes.reshape(-1, c), torch.full((len(s), 4 - c), -1, device="cuda")], 1))
        key, blk, elem, loc, ids = (torch.cat(x) for x in (key, blk, elem, loc, ids))
        visit = (blk << 40) + elem * 8 + loc
        order = torch.argsort(visit)
        order = order[torch.argsort(key[order], stable=True)]
        key, blk, elem, loc, ids = (x[order] for x in (key, blk, elem, loc, ids))
        first = torch.ones(len(key), dtype=torch.bool, device="cuda")
        first[1:] = key[1:] != key[:-1]
        own = first.nonzero()[:, 0]
        paired = torch.zeros(len(own), dtype=torch.bool, device="cuda")
        nxt = torch.clamp(own + 1, max=len(key) - 1)
        paired = (nxt != own) & (key[nxt] == key[own])
        tag_of = {}
        for (kind, data), phys in zip(src.cells, src.physical):
            if kind in ("triangle", "quad") and len(data):
                s = canon[torch.as_tensor(np.asarray(data), device="cuda").long()].sort(-1)[0]
                tag_of[kind] = ((s[:, 0] << 42) | (s[:, 1] << 21) | s[:, 2],
                                torch.as_tensor(np.asarray(phys), device="cuda").long())
        self.groups, area = [], {t: torch.zeros(len(self.conn[t]), dtype=torch.float64, device="cuda") for t in self.types}
        sample = {t: [] for t in self.types}
        corners = ids[own, 3] < 0                                      # triangles
        for c in (3, 4):
            shapes, weights = _face_rule(c, self.P)
            for ob, ot in enumerate(self.types):
                for nb in [-1] + list(range(len(self.types))):
                    sel = (blk[own] == ob) & (corners == (c == 3)) & (paired == (nb >= 0))
                    if nb >= 0:
                        sel &= blk[nxt] == nb
                    o = own[sel]
                    if not len(o):
                        continue
                    g = dict(ot=ot, nt=self.types[nb] if nb >= 0 else None, oc=elem[o])
                    ref_c = torch.stack([torch.nn.functional.pad(_t(_CORNERS[ot])[list(f)], (0, 0, 0, 4 - len(f)))
                                         for f in _FACES[ot]])
                    rc = ref_c[loc[o]][:, :c]                          # (F, c, 3) owner reference corners
                    p = torch.einsum("qc,fcd->fqd", shapes, rc)
                    xyz = self.xyz[ot][g["oc"]]
                    J = torch.einsum("fid,fqir->fqdr", xyz, _basis(ot, 1, p)[1])
                    if c == 3:
                        tu = (rc[:, 1] - rc[:, 0])[:, None].expand_as(p)
                        tv = (rc[:, 2] - rc[:, 0])[:, None].expand_as(p)
                    else:
                        u, v = (shapes[:, 1] + shapes[:, 2])[None, :, None], (shapes[:, 2] + shapes[:, 3])[None, :, None]
                        r0, r1, r2, r3 = (rc[:, k][:, None] for k in range(4))
                        tu = (1 - v) * (r1 - r0) + v * (r2 - r3)
                        tv = (1 - u) * (r3 - r0) + u * (r2 - r1)
                    av = torch.linalg.cross(torch.einsum("fqdr,fqr->fqd", J, tu), torch.einsum("fqdr,fqr->fqd", J, tv))
                    outward = torch.einsum("fqd,fd->fq", av, (torch.einsum("fqi,fid->fqd", _basis(ot, 1, p)[0], xyz).mean(1)
                                                             - xyz.mean(1)))
                    av = av * torch.where(outward >= 0, 1.0, -1.0)[..., None]
                    mag = av.norm(dim=-1)
                    g["n"], g["w"] = av / mag[..., None], weights * mag
                    area[ot].index_add_(0, g["oc"], g["w"].sum(1))
                    self._side(g, "o", ot, g["oc"], p, sample)
                    if nb >= 0:
                        m = nxt[sel]
                        g["nc"] = elem[m]
                        nref = torch.stack([torch.nn.functional.pad(_t(_CORNERS[g["nt"]])[list(f)], (0, 0, 0, 4 - len(f)))
                                            for f in _FACES[g["nt"]]])[loc[m]][:, :c]
                        match = (ids[o][:, :c, None] == ids[m][:, None, :c]).double().argmax(-1)
                        p = torch.einsum("qc,fcd->fqd", shapes, torch.gather(nref, 1, match[..., None].expand(-1, -1, 3)))
                        area[g["nt"]].index_add_(0, g["nc"], g["w"].sum(1))
                        self._side(g, "n", g["nt"], g["nc"], p, sample)
                    else:
                        keys, vals = tag_of["triangle" if c == 3 else "quad"]
                        s, i = keys.sort()
                        g["tag"] = vals[i][torch.searchsorted(s, key[o])]
                    self.groups.append(g)
        self.h, self.Bs = {}, {}
        for t in self.types:
            vol = self.wdet[t].sum(1)
            self.h[t] = torch.maximum(2.0 * vol / area[t], 0.25 * vol ** (1.0 / 3.0) / (self.P + 1))
            s = torch.unique(torch.round(torch.cat(sample[t]), decimals=12), dim=0)
            self.Bs[t] = torch.cat([_basis(t, self.P, _nodes(t, self.P))[0], self.B[t], _basis(t, self.P, s)[0]])

    def _side(self, g, side, t, cells, p, sample):
        flat = torch.unique(torch.round(p.reshape(len(p), -1), decimals=12), dim=0)
        sample[t].append(flat.reshape(-1, 3))
        B, dB = _basis(t, self.P, p)
        g["B" + side] = B
        if self.viscous:
            J = torch.einsum("fid,fqir->fqdr", self.xyz[t][cells], _basis(t, 1, p)[1])
            g["G" + side] = torch.einsum("fqir,fqrd->fqid", dB, torch.linalg.inv(J))

    # ---- physics
    @staticmethod
    def prim(U):
        rho = U[..., 0]
        safe = torch.clamp(rho, min=1e-14)
        vel = U[..., 1:4] / safe[..., None]
        p = (GAMMA - 1.0) * (U[..., 4] - 0.5 * (U[..., 1:4] ** 2).sum(-1) / safe)
        return rho, vel, p

    def flux(self, U, n):
        rho, vel, p = self.prim(U)
        un = (vel * n).sum(-1)
        return torch.cat([(rho * un)[..., None], rho[..., None] * vel * un[..., None] + p[..., None] * n,
                          (un * (U[..., 4] + p))[..., None]], -1)

    def fluxes(self, U):
        eye = torch.eye(3, dtype=U.dtype, device=U.device)
        return torch.stack([self.flux(U, eye[d]) for d in range(3)], -2)

    def hllc(self, UL, UR, n):
        def side(U):
            rho, vel, p = self.prim(U)
            return rho, vel, p, (vel * n).sum(-1), torch.sqrt(torch.clamp(GAMMA * p / torch.clamp(rho, min=1e-14), min=0.0))

        def safe(x, tol=1e-14):
            return torch.where(x.abs() > tol, x, torch.where(x >= 0, tol, -tol).to(x.dtype))

        L, R = side(UL), side(UR)
        FL, FR = self.flux(UL, n), self.flux(UR, n)
        sl, sr = torch.minimum(L[3] - L[4], R[3] - R[4]), torch.maximum(L[3] + L[4], R[3] + R[4])
        aL, aR = L[0] * (sl - L[3]), R[0] * (sr - R[3])
        sm = (R[2] - L[2] + L[3] * aL - R[3] * aR) / safe(aL - aR)

        def star(U, S, s):
            rho, vel, p, un, _ = S
            den = safe(s - sm)
            r = rho * (s - un) / den
            ps = p + rho * (s - un) * (sm - un)
            E = ((s - un) * U[..., 4] - p * un + ps * sm) / den
            return torch.cat([r[..., None], r[..., None] * (vel + (sm - un)[..., None] * n), E[..., None]], -1)

        HL = FL + sl[..., None] * (star(UL, L, sl) - UL)
        HR = FR + sr[..., None] * (star(UR, R, sr) - UR)
        pick = lambda c, a, b: torch.where(c[..., None], a, b)       # noqa: E731
        H = pick(sl >= 0, FL, pick(sm >= 0, HL, pick(sr > 0, HR, FR)))
        good = (L[0] > 0) & (R[0] > 0) & (L[2] > 0) & (R[2] > 0) & torch.isfinite(H).all(-1)
        s = torch.maximum(L[3].abs() + L[4], R[3].abs() + R[4])
        H = pick(good, H, 0.5 * (FL + FR) - 0.5 * s[..., None] * (UR - UL))
        return pick((UL == UR).all(-1), FL, H)

    def vis_vars(self, U):
        rho, vel, p = self.prim(U)
        return torch.cat([vel, (p / torch.clamp(rho, min=1e-14))[..., None]], -1)

    def vis_flux(self, U, grad, mu, kappa):
        vel = self.prim(U)[1]
        G = grad[..., 0:3, :]
        div = G.diagonal(dim1=-2, dim2=-1).sum(-1)
        eye = torch.eye(3, dtype=U.dtype, device=U.device)
        tau = mu[..., None, None] * (G + G.transpose(-1, -2) - (2.0 / 3.0) * div[..., None, None] * eye)
        F = torch.zeros(U.shape[:-1] + (3, 5), dtype=U.dtype, device=U.device)
        F[..., 1:4] = tau.transpose(-1, -2)
        F[..., 4] = torch.einsum("...i,...id->...d", vel, tau) + kappa[..., None] * grad[..., 3, :]
        return F

    def _is(self, tag, role):
        hit = torch.zeros_like(tag, dtype=torch.bool)
        for v in self.roles[role]:
            hit |= tag == v
        return hit[:, None]

    def ghosts(self, g, U):
        """(inviscid ghost state, viscous ghost variables) of boundary faces."""
        if self.far is None:
            return U, self.vis_vars(U)
        far = self.far[self.case_id[g["oc"]]] if self.case_id is not None else self.far.expand(len(U), 5)
        far = far[:, None, :].expand_as(U)
        rho, vel, p = self.prim(U)
        un = (vel * g["n"]).sum(-1, keepdim=True)
        W = torch.cat([rho[..., None], vel, p[..., None]], -1)
        Ww = torch.cat([rho[..., None], vel - 2 * un * g["n"], p[..., None]], -1)
        wall, inlet = self._is(g["tag"], "wall")[..., None], self._is(g["tag"], "inlet")[..., None]
        ghost = _conserved(torch.where(inlet, far, torch.where(wall, Ww, W)))
        v = self.vis_vars(U)
        T = v[..., 3:] if self.wall_T is None else 2.0 * self.wall_T - v[..., 3:]
        v = torch.where(self._is(g["tag"], "no_slip")[..., None], torch.cat([-v[..., :3], T], -1), v)
        sl = torch.cat([v[..., :3] - 2 * (v[..., :3] * g["n"]).sum(-1, keepdim=True) * g["n"], v[..., 3:]], -1)
        v = torch.where(self._is(g["tag"], "slip")[..., None], sl, v)
        return ghost, torch.where(inlet, self.vis_vars(_conserved(far)), v)

    # ---- residual
    def rhs(self, S):
        R = {}
        for t in self.types:
            a = S[t][:, :1]
            Uq = a + torch.einsum("qi,eiv->eqv", self.B[t], S[t] - a)
            F = self.fluxes(Uq) - self.fluxes(a)
            R[t] = torch.einsum("eqid,eqdv,eq->eiv", self.grad[t], F, self.wdet[t])
        vis = {t: self.vis_vars(S[t]) for t in self.types} if self.viscous else None
        lift = {t: torch.zeros(S[t].shape[:2] + (4, 3), dtype=torch.float64, device="cuda") for t in self.types}
        kept = []
        for g in self.groups:
            ot, nt = g["ot"], g["nt"]
            So = S[ot][g["oc"]]
            ao = So[:, :1]
            Uo = ao + torch.einsum("fqi,fiv->fqv", g["Bo"], So - ao)
            if nt:
                Sn = S[nt][g["nc"]]
                an = Sn[:, :1]
                Un = an + torch.einsum("fqi,fiv->fqv", g["Bn"], Sn - an)
            else:
                Un, vg = self.ghosts(g, Uo)
            H = self.hllc(Uo, Un, g["n"])
            w = g["w"][..., None]
            R[ot].index_add_(0, g["oc"], -torch.einsum("fqi,fqv->fiv", g["Bo"], (H - self.flux(ao, g["n"])) * w))
            if nt:
                R[nt].index_add_(0, g["nc"], torch.einsum("fqi,fqv->fiv", g["Bn"], (H - self.flux(an, g["n"])) * w))
            if not self.viscous:
                continue
            vo = torch.einsum("fqi,fim->fqm", g["Bo"], vis[ot][g["oc"]])
            vn = torch.einsum("fqi,fim->fqm", g["Bn"], vis[nt][g["nc"]]) if nt else vg
            jn = 0.5 * torch.einsum("fq,fqm,fqd->fqmd", g["w"], vn - vo, g["n"])
            lo = torch.einsum("fij,fqj,fqmd->fimd", self.minv[ot][g["oc"]], g["Bo"], jn)
            lift[ot].index_add_(0, g["oc"], lo)
            ln = None
            if nt:
                ln = torch.einsum("fij,fqj,fqmd->fimd", self.minv[nt][g["nc"]], g["Bn"], jn)
                lift[nt].index_add_(0, g["nc"], ln)
            kept.append((Uo, Un, lo, ln))
        if self.viscous:
            for t in self.types:
                Uq = torch.einsum("qi,eiv->eqv", self.B[t], S[t])
                grad = torch.einsum("eim,eqid->eqmd", vis[t], self.grad[t]) + torch.einsum("qi,eimd->eqmd", self.B[t], lift[t])
                F = self.vis_flux(Uq, grad, self.mu[t][:, None].expand(Uq.shape[:2]), self.kappa[t][:, None].expand(Uq.shape[:2]))
                R[t] -= torch.einsum("eqid,eqdv,eq->eiv", self.grad[t], F, self.wdet[t])
            for g, (Uo, Un, lo, ln) in zip(self.groups, kept):
                ot, nt = g["ot"], g["nt"]
                mu, ka = (x[ot][g["oc"]][:, None].expand(Uo.shape[:2]) for x in (self.mu, self.kappa))
                raw = torch.einsum("fim,fqid->fqmd", vis[ot][g["oc"]], g["Go"])
                F = self.vis_flux(Uo, raw + self.br2 * torch.einsum("fqi,fimd->fqmd", g["Bo"], lo), mu, ka)
                if nt:
                    raw = torch.einsum("fim,fqid->fqmd", vis[nt][g["nc"]], g["Gn"])
                    F = 0.5 * (F + self.vis_flux(Un, raw + self.br2 * torch.einsum("fqi,fimd->fqmd", g["Bn"], ln), mu, ka))
                Fn = torch.einsum("fqdv,fqd->fqv", F, g["n"])
                if not nt and self.far is not None:
                    Fn[..., 4] = torch.where(self._is(g["tag"], "wall"), 0.0, Fn[..., 4])
                Fn = Fn * g["w"][..., None]
                R[ot].index_add_(0, g["oc"], torch.einsum("fqi,fqv->fiv", g["Bo"], Fn))
                if nt:
                    R[nt].index_add_(0, g["nc"], -torch.einsum("fqi,fqv->fiv", g["Bn"], Fn))
        return {t: torch.einsum("eij,ejv->eiv", self.minv[t], R[t]) for t in self.types}

    # ---- time
    def stable_dt(self, S, cfl=0.3):
        df, worst = 2 * self.P + 1, 1e-12
        for t in self.types:
            rho, vel, p = self.prim(S[t])
            rho, p = torch.clamp(rho, min=1e-14), torch.clamp(p, min=1e-14)
            rate = df * (vel.norm(dim=-1) + torch.sqrt(GAMMA * p / rho)).amax(1) / self.h[t]
            if self.viscous:
                rm = torch.clamp(rho.mean(1), min=0.1)
                diff = torch.maximum((4.0 / 3.0) * self.mu[t] / rm, self.kappa[t] / (rm * GAMMA / (GAMMA - 1.0)))
                rate = rate + 2.0 * self.br2 * df ** 2 * diff / torch.clamp(self.h[t], min=0.01) ** 2
            worst = max(worst, float(rate.max()))
        return min(max(cfl / worst, 1e-7), 1e-3)

    def limit(self, S, floor=1e-10, relative=0.05):
        out = {}
        for t in self.types:
            U = S[t]
            Uq = torch.einsum("qi,eiv->eqv", self.B[t], U)
            mean = torch.einsum("eqv,eq->ev", Uq, self.wdet[t]) / self.wdet[t].sum(1)[:, None]
            rm, _, pm = self.prim(mean)
            rf, pf = torch.clamp(relative * rm, min=floor), torch.clamp(relative * pm, min=floor)
            dev = torch.einsum("qi,eiv->eqv", self.Bs[t], U) - mean[:, None]
            low = (mean[:, None, 0] + dev[..., 0]).amin(1)
            up = torch.where(low < rf, (rm - rf) / torch.clamp(rm - low, min=1e-30), 1.0).clamp(0.0, 1.0)
            ok = lambda th: self.prim(mean[:, None] + th[:, None, None] * dev)[2].amin(1) >= pf      # noqa: E731
            lo, hi = torch.zeros_like(up), up.clone()
            for _ in range(30):
                mid = 0.5 * (lo + hi)
                good = ok(mid)
                lo, hi = torch.where(good, mid, lo), torch.where(good, hi, mid)
            theta = torch.where(ok(up), up, lo)
            out[t] = mean[:, None] + theta[:, None, None] * (U - mean[:, None])
        return out

    def step(self, S, dt, limited):
        cur, valid, rho_min, p_min = S, True, math.inf, math.inf
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)):
            R = self.rhs(cur)
            cur = {t: a * S[t] + b * (cur[t] + dt * R[t]) for t in self.types}
            cur = self.limit(cur) if limited else cur
            for U in cur.values():
                rho, _, p = self.prim(U)
                rho_min, p_min = min(rho_min, float(rho.min())), min(p_min, float(p.min()))
                valid &= bool(torch.isfinite(U).all())
        return cur, valid and rho_min >= 1e-7 and p_min >= 1e-7, rho_min, p_min


class _PlainSource:
    """The Air-11 source: Newton on rho - rho0 - dt w(rho, T(rho)) with the analytic Jacobian of w."""

    def __init__(self, coupler):
        sp, rx = AIR11_SPECIES, AIR11_REACTIONS
        ns, nr = len(sp), len(rx)
        self.W = _t([s.molar_mass for s in sp])
        self.range = _t([[s.poly.t_low, s.poly.t_mid, s.poly.t_high] for s in sp])
        self.fit = _t([[s.poly.coeffs_low, s.poly.coeffs_high] for s in sp])
        f, r, alpha = np.zeros((nr, ns)), np.zeros((nr, ns)), np.zeros((nr, ns))
        for i, x in enumerate(rx):
            for s, c in x.reactants:
                f[i, s] += c
            for s, c in x.products:
                r[i, s] += c
            if x.third_body:
                alpha[i] = [0.0 if s.name == "e-" else 1.0 for s in sp]
                for s, e in x.efficiencies:
                    alpha[i, s] = e
        self.nf, self.nr, self.alpha = _t(f), _t(r), _t(alpha)
        self.third = torch.tensor([bool(x.third_body) for x in rx], device="cuda")
        self.arr = [_t([getattr(x, k) for x in rx]) for k in ("A", "b", "theta")]
        self.Ru, self.c = 8.31446261815324, coupler

    def _fits(self, T):
        Tc = torch.minimum(torch.maximum(T[:, None], self.range[:, 0]), self.range[:, 2])
        a = torch.where((Tc < self.range[:, 1])[..., None], self.fit[:, 0], self.fit[:, 1])
        cp = a[..., 0] + Tc * (a[..., 1] + Tc * (a[..., 2] + Tc * (a[..., 3] + Tc * a[..., 4])))
        h = (a[..., 0] + Tc * (a[..., 1] / 2 + Tc * (a[..., 2] / 3 + Tc * (a[..., 3] / 4 + Tc * a[..., 4] / 5)))
             + a[..., 5] / Tc)
        s = (a[..., 0] * torch.log(Tc) + Tc * (a[..., 1] + Tc * (a[..., 2] / 2 + Tc * (a[..., 3] / 3 + Tc * a[..., 4] / 4)))
             + a[..., 6])
        return cp, h, s

    def _energy(self, T):
        cp, h, _ = self._fits(T)
        return (h - 1.0) * (self.Ru * T[:, None] / self.W), (cp - 1.0) * (self.Ru / self.W)

    def temperature(self, rho, e, T, n):
        Y = torch.clamp(rho, min=0.0) / torch.clamp(rho.sum(1), min=1e-14)[:, None]
        for _ in range(n):
            es, cv = self._energy(T.clamp(50.0, 50000.0))
            d = -((Y * es).sum(1) - e) / torch.clamp((Y * cv).sum(1), min=1e-5)
            T = (T + torch.minimum(torch.maximum(d, -0.5 * T), 0.5 * T)).clamp(100.0, 50000.0)
        return T

    def rates(self, rho, T):
        A, b, theta = self.arr
        raw = rho / self.W
        C = torch.clamp(raw, min=0.0)
        Tg = torch.clamp(T, min=10.0)[:, None]
        kf = A * Tg ** b * torch.exp(-theta / Tg)
        _, h, s = self._fits(Tg[:, 0])
        nu = self.nr - self.nf
        kc = torch.exp(-((h - s) @ nu.T).clamp(-700.0, 700.0)) * (101325.0 / (self.Ru * Tg)) ** nu.sum(1)
        kr = kf / torch.clamp(kc, min=1e-300)
        logC = torch.log(torch.clamp(C, min=1e-100))
        lf, lr = logC @ self.nf.T, logC @ self.nr.T
        F, B = kf * torch.exp(lf.clamp(-700, 700)), kr * torch.exp(lr.clamp(-700, 700))
        coll = torch.where(self.third, C @ self.alpha.T, 1.0)
        w = (((F - B) * coll) @ nu) * self.W
        dC = torch.where(raw > 0, 1.0, torch.where(raw == 0, 0.5, 0.0)) / self.W
        dlog = torch.where(C > 1e-100, 1.0, torch.where(C == 1e-100, 0.5, 0.0)) * dC / torch.clamp(C, min=1e-100)
        Fk, Bk = F * (lf.abs() < 700), B * (lr.abs() < 700)
        dq = (Fk[..., None] * self.nf - Bk[..., None] * self.nr) * dlog[:, None] * coll[..., None]
        dq = dq + (F - B)[..., None] * torch.where(self.third[:, None], self.alpha, 0.0) * dC[:, None]
        J = self.W[:, None] * torch.einsum("rs,nrj->nsj", nu, dq)
        total = rho.sum(1)
        S = torch.clamp(total, min=1e-14)[:, None]
        Y, sw = torch.clamp(rho, min=0.0) / S, w.sum(1, keepdim=True)
        pos = torch.where(rho > 0, 1.0, torch.where(rho == 0, 0.5, 0.0))
        dY = torch.diag_embed(pos / S) - (Y / S * (total > 1e-14)[:, None])[..., None]
        return w - Y * sw, J - dY * sw[..., None] - Y[..., None] * J.sum(1)[:, None]

    def __call__(self, U, dt):
        c, u = self.c, U.reshape(-1, U.shape[-1])
        rho_t = torch.clamp(u[:, 0], min=1e-14)
        rs = torch.clamp(u[:, 5:16], min=0.0)
        rs = rs * (rho_t / torch.clamp(rs.sum(1), min=1e-20))[:, None] * c.rho_ref
        es = torch.clamp(u[:, 4] / rho_t - 0.5 * (u[:, 1:4] ** 2).sum(1) / rho_t ** 2, min=1e-4)
        T = self.temperature(rs, es * c.e_ref, torch.clamp((GAMMA - 1.0) * es * c.T_ref, min=200.0), 8)
        rho0 = torch.clamp(rs, min=1e-20)
        e = (rho0 / rho0.sum(1, keepdim=True) * self._energy(T)[0]).sum(1)
        rho, step, eye = rho0, dt * c.t_ref, torch.eye(11, dtype=torch.float64, device="cuda")
        for _ in range(c.max_newton_iters):
            w, J = self.rates(rho, T)
            rho = torch.clamp(rho + torch.linalg.solve_ex(eye - step * J, -(rho - rho0 - step * w))[0], min=0.0)
            T = self.temperature(rho, e, T, 10)
        rho = rho * (rho0.sum(1) / rho.sum(1))[:, None] / c.rho_ref
        out = u.clone()
        out[:, 5:16] = rho * (rho_t / rho.sum(1))[:, None]
        return out.reshape(U.shape)


def exact(case, seed):
    family = case["family"]
    if family == "source":
        return _PlainSource(_coupler(case["iterations"]))(_hot_nodes(case, seed), SOURCE_DT)
    if family == "reacting" or case.get("limiter") == "mood":
        return None                                  # MOOD: see the head of this file
    P, ids, far, prandtl = case["degree"], None, None, 0.72
    if family == "cylinders":
        parts = _ensemble(case)
        src, _ = meshgen.union([p[0] for p in parts])
        ids = torch.cat([torch.full((len(p[0].cells[0][1]),), k) for k, p in enumerate(parts)]).cuda()
        plain = _Plain(src, P, mu=[p[2] for p in parts], far=_t(np.stack([p[1] for p in parts])), case_id=ids)
    elif family == "sphere":
        far = np.array([1.0, wl.SPHERE_MACH * math.sqrt(GAMMA), 0.0, 0.0, 1.0])
        plain = _Plain(_sphere_source(case), P, mu=far[1] / wl.SPHERE_RE, far=_t(far),
                       wall_T=wl.SPHERE_T_WALL / wl.SPHERE_T_INF)
    elif family == "taylor":
        plain = _Plain(wl.tgv_mesh(case["n"]), P, prandtl=0.71, mu=1.0 / 1600.0)
    else:
        src = meshgen.hybrid_box((case["n"],) * 3, hi=(10.0,) * 3, jitter=0.1, seed=0)
        plain = _Plain(src, P, mu=0.0 if family == "vortex" else 1e-2)
    S = {}
    for t in plain.types:
        xyz = torch.einsum("ni,eid->end", _basis(t, 1, _nodes(t, P))[0], plain.xyz[t])
        S[t] = _conserved(_primitive(case, t, xyz, seed, ids))
    if family == "rhs":
        return plain.rhs(S)
    out, valid, rho_min, p_min = plain.step(S, plain.stable_dt(S), case.get("limiter") == "positivity")
    out["valid"], out["minima"] = torch.tensor([int(valid)], dtype=torch.int32), _t([rho_min, p_min])
    return out
