"""Performance cases of the field solver, each one pass through the public entry points.

``listed()`` holds the fixed cases, ``draw(rng)`` one more case of the same ranges,
``prepare(case, seed)`` what a program has in hand before the call, ``run(state)`` one
pass, ``work(case)`` the bytes and operations that a pass cannot do without and
``exact(case, seed)`` the results as direct sums in 64 bits in plain torch.

Kinds of case (``kind``):

* ``sim``     one ``ElectrostaticSimulation.step`` (direct sums up to 1000 particles, the
              Coulomb FMM of order 4 with leaves of 32 above);
* ``walk``    a fresh tree and the Barnes-Hut walk at its own particles;
* ``direct``  ``direct_field`` at some of the sources (the solver's accuracy check);
* ``fmm``     a fresh tree and its FMM field;
* ``grad``    ``fmm_energy`` or ``fmm_field`` and the backward to positions and charges;
* ``fmm_at``  a fresh tree and the FMM at other points;
* ``panels``  one product of the electrode solver: new charges on a kept tree, ``fmm_at``;
* ``strip``   line charges between grounded plates.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from tree_d_3d_b200 import FlatQuadtree, GroundedStripField, Quad, direct_field
from tree_d_3d_b200.autograd import fmm_energy, fmm_field
from tree_d_3d_b200.electrodes import PanelSums
from tree_d_3d_b200.simulation import ElectrostaticSimulation

DEV = "cuda"
ROOT = (0.0, 0.0, 1.0)
#: softening of the point-charge cases; line charges are summed unsoftened
EPS = 1e-3
#: most directed pairs that exact() sums
EXACT_PAIRS = 1.05e12


# --------------------------------------------------------------------------- the cases
def listed() -> list:
    return [
        # a step of a small interactive simulation: direct sums, bound by latency
        {"name": "sim_direct_1k", "kind": "sim", "n": 1000, "precision": "fp64"},
        # the workload table's first line: 5000 uniform charges, Barnes-Hut
        {"name": "walk_5k", "kind": "walk", "n": 5000, "dist": "uniform", "kernel": "coulomb",
         "theta": 0.5, "precision": "fp64"},
        # the accuracy check that goes with a field solve: sampled particles, every source
        {"name": "direct_log_4096x200k", "kind": "direct", "n": 200_000, "m": 4096,
         "dist": "gaussian", "kernel": "log"},
        # line charges of a 2D Gaussian beam, the plain FP64 solve
        {"name": "fmm_log_200k", "kind": "fmm", "n": 200_003, "dist": "gaussian",
         "kernel": "log", "order": 12, "leaf": 8, "theta": 0.5, "precision": "fp64"},
        # the headline workload: 1M clustered line charges, mixed precision, with backward
        {"name": "grad_log_1M_mixed", "kind": "grad", "n": 1_000_000, "dist": "mixture",
         "kernel": "log", "order": 12, "leaf": 8, "theta": 0.5, "precision": "mixed",
         "loss": "energy"},
        # Barnes-Hut at 1M clustered charges
        {"name": "walk_1M", "kind": "walk", "n": 1_000_000, "dist": "mixture",
         "kernel": "coulomb", "theta": 0.5, "precision": "fp64"},
        # the high-order point-charge solve at 1M clustered charges, FP64
        {"name": "fmm_coulomb_1M_p12", "kind": "fmm", "n": 1_000_000, "dist": "mixture",
         "kernel": "coulomb", "order": 12, "leaf": 8, "theta": 0.5, "precision": "fp64"},
        # the differentiation workload: 100k point charges, potential and field in the loss
        {"name": "grad_coulomb_100k_mixed", "kind": "grad", "n": 99_991, "dist": "uniform",
         "kernel": "coulomb", "order": 12, "leaf": 8, "theta": 0.5, "precision": "mixed",
         "loss": "field"},
        # a step of the large simulation: 1M particles, Coulomb FMM at the defaults
        {"name": "sim_fmm_1M", "kind": "sim", "n": 1_000_000, "precision": "fp64"},
        # the field of a clustered source set at as many points off the sources
        {"name": "fmm_at_log_500k_mixed", "kind": "fmm_at", "n": 500_000, "m": 499_979,
         "dist": "mixture", "kernel": "log", "order": 12, "leaf": 8, "theta": 0.5,
         "precision": "mixed"},
        # an iteration of the electrode solver: order 32 on panel nodes
        {"name": "panels_48k", "kind": "panels", "n": 48_000, "precision": "fp64"},
        # a beam between grounded plates, close pairs softened
        {"name": "strip_50k", "kind": "strip", "n": 50_001},
    ]


def _log_uniform(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["sim", "walk", "direct", "fmm", "fmm", "grad", "grad", "fmm_at",
                       "panels", "strip"])
    precision = rng.choice(["fp64", "mixed"])
    kernel = rng.choice(["log", "coulomb"])
    dist = rng.choice(["uniform", "gaussian", "mixture"])
    theta = rng.choice([0.4, 0.5, 0.6])
    if kind == "sim":
        return {"kind": kind, "n": _log_uniform(rng, 200, 500_000), "precision": precision}
    if kind == "strip":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 80_000)}
    if kind == "panels":
        return {"kind": kind, "n": 4 * _log_uniform(rng, 500, 20_000), "precision": precision}
    if kind == "direct":
        return {"kind": kind, "n": _log_uniform(rng, 2000, 200_000),
                "m": _log_uniform(rng, 64, 8192), "dist": dist, "kernel": kernel}
    if kind == "walk":
        return {"kind": kind, "n": _log_uniform(rng, 2000, 1_000_000), "dist": dist,
                "kernel": kernel, "theta": rng.choice([0.4, 0.5, 0.6, 0.7]),
                "precision": precision}
    order = rng.randint(4, 16)
    case = {"kind": kind, "n": 0, "dist": dist, "kernel": kernel, "order": order,
            "leaf": rng.choice([8, 16, 32]), "theta": theta, "precision": precision}
    # point charges at high order are the dear ones: fewer particles
    most = 1_000_000 if kernel == "log" else 500_000 if order <= 10 else 150_000
    if theta < 0.5:
        most //= 2
    if kind == "fmm":
        return dict(case, n=_log_uniform(rng, 2000, most))
    if kind == "fmm_at":
        return dict(case, n=_log_uniform(rng, 2000, most), m=_log_uniform(rng, 2000, most))
    loss = rng.choice(["energy", "field"])
    most = min(most, 250_000) if loss == "field" or kernel == "coulomb" else most
    return dict(case, n=_log_uniform(rng, 2000, most), loss=loss)


# --------------------------------------------------------------------------- the inputs
def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _uniform(g, *shape):
    return 2 * torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64) - 1


def _signs(g, n: int):
    return torch.where(torch.rand(n, generator=g, device=DEV) < 0.5, -1.0, 1.0).double()


def _positions(g, n: int, dist: str) -> torch.Tensor:
    """(2, n) points inside (-1, 1)^2; what falls outside is drawn again."""
    if dist == "uniform":
        return _uniform(g, 2, n)
    centres = 0.8 * _uniform(g, 2, 8)
    sigmas = torch.linspace(0.02, 0.2, 8, device=DEV, dtype=torch.float64)
    parts, have = [], 0
    while have < n:
        k = int(1.3 * (n - have)) + 1024
        if dist == "gaussian":
            pts = 0.3 * _normal(g, 2, k)
        elif dist == "protons":
            pts = 0.1 * _normal(g, 2, k)
        else:
            label = torch.randint(0, 8, (k,), generator=g, device=DEV)
            pts = centres[:, label] + sigmas[label] * _normal(g, 2, k)
        pts = pts[:, (pts.abs() < 1).all(0)]
        parts.append(pts)
        have += pts.shape[1]
    return torch.cat(parts, dim=1)[:, :n].contiguous()


def _panels(n: int, g):
    """Nodes along three closed curves and a segment (n / 4 each, turned and moved a little
    by the seed), the midpoints and every fifth node as targets, the latter without their
    own node."""
    k = n // 4
    shift = (0.02 * torch.rand(8, generator=g, device=DEV, dtype=torch.float64)).tolist()
    t = np.linspace(0.0, 2 * np.pi, k, endpoint=False) + 50 * shift[0]
    curves = [np.stack((0.3 * np.cos(t) - 0.4 + shift[1], 0.3 * np.sin(t) + 0.1 + shift[2])),
              np.stack((0.2 * np.cos(t) + 0.45 + shift[3], 0.25 * np.sin(t) - 0.2 + shift[4])),
              np.stack((0.1 * np.cos(t) + 0.1 + shift[5], 0.1 * np.sin(t) + 0.6 + shift[6])),
              np.stack((np.linspace(-0.9, 0.9, k), np.full(k, -0.7 - shift[7])))]
    nodes = np.concatenate(curves, axis=1)
    mids = 0.5 * (nodes[:, :-1] + nodes[:, 1:])[:, ::2]
    on_node = np.arange(0, nodes.shape[1], 5)
    targets = np.concatenate((mids, nodes[:, on_node]), axis=1)
    exclude = np.concatenate((np.full(mids.shape[1], -1), on_node)).astype(np.int64)
    return (torch.tensor(nodes, device=DEV), torch.tensor(targets, device=DEV),
            torch.tensor(exclude, device=DEV))


def _inputs(case: dict, seed: int) -> dict:
    g = _generator(seed)
    kind, n = case["kind"], case["n"]
    if kind == "sim":
        return {"pos": _positions(g, n, "protons"), "vel": 0.1 * _normal(g, 2, n),
                "q": torch.ones(n, device=DEV, dtype=torch.float64)}
    if kind == "strip":
        width = 3.0
        x = width * (0.01 + 0.98 * (0.5 * _uniform(g, n) + 0.5))
        return {"width": width, "softening": 0.004, "k_e": 1.0,
                "pos": torch.stack((x, _normal(g, n))), "q": _signs(g, n)}
    if kind == "panels":
        nodes, targets, exclude = _panels(n, g)
        return {"pos": nodes, "targets": targets, "exclude": exclude, "q": _normal(g, n)}
    x = {"pos": _positions(g, n, case["dist"])}
    # the differentiation workload has normal charges, the others +-1
    x["q"] = _normal(g, n) if kind == "grad" and case["dist"] == "uniform" else _signs(g, n)
    if kind == "direct":
        idx = torch.randperm(n, generator=g, device=DEV)[: case["m"]]
        x |= {"exclude": idx, "targets": x["pos"][:, idx].contiguous()}
    elif kind == "walk":
        x["exclude"] = torch.arange(n, device=DEV)
    elif kind == "fmm_at":
        x["targets"] = _uniform(g, 2, case["m"])
    elif kind == "grad":
        x |= {"w": _normal(g, n), "e": _normal(g, 2, n)}
    return x


def _eps(case: dict) -> float:
    return EPS if case.get("kernel", "coulomb") == "coulomb" else 0.0


def _simulation_of(case: dict) -> dict:
    """A cloud of unit total charge and a small step: the state barely moves in a pass."""
    return {"k_e": 1.0 / case["n"], "dt": 1e-6, "B_z": 1.0, "softening": EPS}


def prepare(case: dict, seed: int) -> dict:
    x = _inputs(case, seed)
    state = {"case": case, **x}
    if case["kind"] == "sim":
        state["sim"] = ElectrostaticSimulation(
            positions=x["pos"], velocities=x["vel"], charges=x["q"], bounds=Quad(*ROOT),
            theta=0.5, precision=case["precision"],
            absorbing_walls={"x_min": -1.0, "x_max": 1.0, "y_min": -1.0, "y_max": 1.0},
            **_simulation_of(case))
    elif case["kind"] == "strip":
        state["strip"] = GroundedStripField(x["width"], k_e=x["k_e"], softening=x["softening"])
    elif case["kind"] == "panels":
        # the solver's iterations: the tree and the target plan are made by the first product
        state["sums"] = PanelSums(x["pos"], x["targets"], exclude=x["exclude"],
                                  precision=case["precision"])
        state["sums"](torch.ones_like(x["q"]))
    return state


# --------------------------------------------------------------------------- one pass
def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "sim":
        sim = state["sim"]
        sim.step()
        return sim.positions, sim.velocities, sim.forces
    if kind == "strip":
        return state["strip"].field_at_charges(state["pos"], state["q"])
    if kind == "panels":
        return state["sums"](state["q"])
    if kind == "direct":
        return direct_field(state["targets"], state["pos"], state["q"], softening=_eps(case),
                            exclude=state["exclude"], kernel=case["kernel"])
    if kind == "walk":
        tree = FlatQuadtree(state["pos"], state["q"], Quad(*ROOT), kernel=case["kernel"],
                            precision=case["precision"])
        return tree.evaluate(state["pos"], exclude=state["exclude"], theta=case["theta"],
                             softening=_eps(case))
    if kind == "grad":
        options = {"kernel": case["kernel"], "order": case["order"], "theta": case["theta"],
                   "softening": _eps(case), "leaf_capacity": case["leaf"],
                   "precision": case["precision"]}
        pos = state["pos"].detach().requires_grad_(True)
        q = state["q"].detach().requires_grad_(True)
        if case["loss"] == "energy":
            energy = fmm_energy(pos, q, Quad(*ROOT), **options)
            energy.backward()
            return energy.detach(), pos.grad, q.grad
        phi, field = fmm_field(pos, q, Quad(*ROOT), **options)
        ((state["w"] * phi).sum() + (state["e"] * field).sum()).backward()
        return phi.detach(), field.detach(), pos.grad, q.grad
    tree = FlatQuadtree(state["pos"], state["q"], Quad(*ROOT), kernel=case["kernel"],
                        order=case["order"], leaf_capacity=case["leaf"],
                        precision=case["precision"])
    if kind == "fmm":
        return tree.fmm(theta=case["theta"], softening=_eps(case))
    return tree.fmm_at(state["targets"], theta=case["theta"], softening=_eps(case))


# --------------------------------------------------------------------------- the work
def _expansion_flops(kernel: str, order: int) -> float:
    """One translation between cells: 8 (p + 1)^2 for complex expansions, the products of
    two triangles of Cartesian coefficients otherwise."""
    if kernel == "log":
        return 8.0 * (order + 1) ** 2
    return 2.0 * math.comb(order + 4, 4)


def _fmm_flops(n: int, kernel: str, order: int, leaf: int, theta: float) -> float:
    """Translations and near pairs of a balanced tree: cells hold about leaf / 2 particles,
    each takes about 7 / theta^2 translations and 9 / (2 theta)^2 near leaves."""
    cells = 4 / 3 * n / (leaf / 2)
    return (cells * 7 / theta**2 * _expansion_flops(kernel, order)
            + n * 9 / (2 * theta) ** 2 * leaf / 2 * 12)


def work(case: dict) -> dict:
    kind, n = case["kind"], case["n"]
    if kind == "direct":
        return {"bytes": 8.0 * (3 * n + 6 * case["m"]), "flops": 12.0 * n * case["m"]}
    if kind == "sim":
        flops = 12.0 * n * n if n <= 1000 else _fmm_flops(n, "coulomb", 4, 32, 0.5)
        return {"bytes": 8.0 * 13 * n, "flops": flops}
    if kind == "walk":
        # cells and particles that a target meets, 20 operations each
        return {"bytes": 8.0 * 7 * n, "flops": 20.0 * n * 20 / case["theta"] ** 2}
    if kind == "panels":
        m = 0.7 * n
        return {"bytes": 8.0 * (3 * n + 6 * m), "flops": _fmm_flops(n, "log", 32, 16, 0.5)}
    if kind == "strip":
        return {"bytes": 8.0 * 6 * n, "flops": _fmm_flops(2 * n, "log", 14, 32, 0.5)}
    flops = _fmm_flops(n, case["kernel"], case["order"], case["leaf"], case["theta"])
    if kind == "fmm":
        return {"bytes": 8.0 * 6 * n, "flops": flops}
    if kind == "fmm_at":
        most = max(n, case["m"])
        flops = _fmm_flops(most, case["kernel"], case["order"], case["leaf"], case["theta"])
        return {"bytes": 8.0 * (3 * n + 5 * case["m"]), "flops": flops}
    return {"bytes": 8.0 * (12 if case["loss"] == "field" else 6) * n, "flops": 2 * flops}


# --------------------------------------------------------------------------- 64-bit sums
def _radial(r2, kernel: str, eps: float):
    """(g, h, sg, sh) of squared distances, in place of r2: sg g is the potential and sh h
    the factor of the field sh h d; a log of an infinite distance is left to the caller."""
    if kernel == "log":
        return torch.log(r2), r2.reciprocal_(), -1.0, 2.0
    g = r2.add_(eps * eps).rsqrt_()
    return g, g * g * g, 1.0, 1.0


def _self_sums(pos, q, kernel: str, eps: float):
    """phi (n,) and field (2, n) of the sources at themselves, each pair once: tiles of
    T x T distances, both directions summed by products with [q] and [q, q x, q y]
    (coordinates from the row tile's first point)."""
    n, T = pos.shape[1], 3072
    phi = torch.zeros(n, dtype=torch.float64, device=pos.device)
    field = torch.zeros_like(pos)
    for a in range(0, n, T):
        i = slice(a, min(a + T, n))
        xi, yi = pos[0, i, None], pos[1, i, None]
        origin = pos[:, a:a + 1]
        ci = torch.stack((q[i], q[i] * (pos[0, i] - origin[0]), q[i] * (pos[1, i] - origin[1])), 1)
        for b in range(a, n, T):
            j = slice(b, min(b + T, n))
            r2 = (xi - pos[0, j]).square_()
            dy = yi - pos[1, j]
            r2.addcmul_(dy, dy)
            if a == b:
                r2.fill_diagonal_(math.inf)
            g, h, sg, sh = _radial(r2, kernel, eps)
            if a == b:
                g.fill_diagonal_(0)
            u = pos[:, j] - origin
            cj = torch.stack((q[j], q[j] * u[0], q[j] * u[1]), 1)
            phi[i] += sg * (g @ q[j])
            s = sh * (h @ cj)
            field[:, i] += (pos[:, i] - origin) * s[:, 0] - s[:, 1:].T
            if a != b:
                phi[j] += sg * (q[i] @ g)
                s = sh * (h.T @ ci)
                field[:, j] += u * s[:, 0] - s[:, 1:].T
    return phi, field


def _target_sums(targets, exclude, pos, q, kernel: str, eps: float):
    """phi (m,) and field (2, m) at ``targets``; exclude[i] a source left out (-1: none)."""
    m, n = targets.shape[1], pos.shape[1]
    S, T = 4096, 4096
    phi = torch.zeros(m, dtype=torch.float64, device=pos.device)
    field = torch.zeros_like(targets)
    for a in range(0, m, T):
        i = slice(a, min(a + T, m))
        rows = torch.arange(i.stop - a, device=pos.device)
        for b in range(0, n, S):
            j = slice(b, min(b + S, n))
            dx = targets[0, i, None] - pos[0, j]
            dy = targets[1, i, None] - pos[1, j]
            r2 = dx.square().addcmul_(dy, dy)
            if exclude is not None:
                hit = (exclude[i] >= b) & (exclude[i] < j.stop)
                own = rows[hit], exclude[i][hit] - b
                r2[own] = math.inf
            g, h, sg, sh = _radial(r2, kernel, eps)
            if exclude is not None:
                g[own] = 0
            phi[i] += sg * (g @ q[j])
            field[0, i] += sh * (dx.mul_(h) @ q[j])
            field[1, i] += sh * (dy.mul_(h) @ q[j])
    return phi, field


def _field_loss_gradients(pos, q, w, e, kernel: str, eps: float):
    """phi, field and the gradients of sum w phi + sum e . field to pos and q."""
    n, T = pos.shape[1], 4096
    z = torch.zeros(n, dtype=torch.float64, device=pos.device)
    phi, field, gpos, gq = z.clone(), torch.zeros_like(pos), torch.zeros_like(pos), z.clone()
    for a in range(0, n, T):
        i = slice(a, min(a + T, n))
        for b in range(0, n, T):
            j = slice(b, min(b + T, n))
            dx = pos[0, i, None] - pos[0, j]
            dy = pos[1, i, None] - pos[1, j]
            r2 = dx.square().addcmul_(dy, dy)
            if a == b:
                r2.fill_diagonal_(math.inf)
            g, h, sg, sh = _radial(r2.clone(), kernel, eps)
            if a == b:
                g.fill_diagonal_(0)
            g, h = sg * g, sh * h
            # d (h d) / d d = h I - k d d^T
            k = r2.square().reciprocal_().mul_(4) if kernel == "log" else \
                r2.add_(eps * eps).pow_(-2.5).mul_(3)
            s = g @ torch.stack((q[j], w[j]), 1)
            phi[i] += s[:, 0]
            gq[i] += s[:, 1]
            hx, hy = h * dx, h * dy
            sx = hx @ torch.stack((q[j], w[j], e[0, j]), 1)
            sy = hy @ torch.stack((q[j], w[j], e[1, j]), 1)
            del g, hx, hy
            ei, qi, wi = e[:, i], q[i], w[i]
            field[0, i] += sx[:, 0]
            field[1, i] += sy[:, 0]
            gq[i] -= sx[:, 2] + sy[:, 2]
            gpos[0, i] -= wi * sx[:, 0] + qi * sx[:, 1]
            gpos[1, i] -= wi * sy[:, 0] + qi * sy[:, 1]
            if a == b:  # the self pairs: infinite distances, finite differences of zero
                k.fill_diagonal_(0)
            cols = torch.stack((q[j], e[0, j], e[1, j]), 1)
            jxx = (h - k * dx * dx) @ cols
            jxy = (k * dx * dy).neg_() @ cols
            jyy = (h - k * dy * dy) @ cols
            gpos[0, i] += jxx[:, 0] * ei[0] + jxy[:, 0] * ei[1] - qi * (jxx[:, 1] + jxy[:, 2])
            gpos[1, i] += jxy[:, 0] * ei[0] + jyy[:, 0] * ei[1] - qi * (jxy[:, 1] + jyy[:, 2])
    return phi, field, gpos, gq


def _drift(pos, vel, angle, dt):
    """The exact turn of a uniform magnetic field over dt: new positions and velocities."""
    c, s = math.cos(angle), math.sin(angle)
    a = s / angle
    b = (1 - c) / angle
    turned = torch.stack((c * vel[0] + s * vel[1], c * vel[1] - s * vel[0]))
    return pos + dt * torch.stack((a * vel[0] + b * vel[1], a * vel[1] - b * vel[0])), turned


def _exact_step(x: dict, case: dict):
    p = _simulation_of(case)
    pos, vel, q, dt = x["pos"], x["vel"], x["q"], p["dt"]

    def force(at):
        return p["k_e"] * q * _self_sums(at, q, "coulomb", p["softening"])[1]

    vel = vel + 0.5 * dt * force(pos)
    pos, vel = _drift(pos, vel, p["B_z"] * dt, dt)
    f = force(pos)
    vel = vel + 0.5 * dt * f
    return pos, vel, f + p["B_z"] * q * torch.stack((vel[1], -vel[0]))


def _exact_strip(x: dict):
    """Green's function between the plates, with every charge's own image force and the
    softening of close pairs."""
    pos, q, width, soft = x["pos"], x["q"], x["width"], x["softening"]
    n, T = pos.shape[1], 2048
    scale = math.pi / (2 * width)
    z = torch.complex(pos[0], pos[1])
    phi = torch.zeros(n, dtype=torch.float64, device=pos.device)
    field = torch.zeros_like(pos)
    for a in range(0, n, T):
        i = slice(a, min(a + T, n))
        for b in range(0, n, T):
            j = slice(b, min(b + T, n))
            d = z[i, None] - z[j]
            dx, dy = d.real.contiguous(), d.imag.contiguous()
            sx = z[i, None].real + z[j].real
            # |sin(scale (x + i y))|^2 = sin^2 + sinh^2, cot = (sin cos - i sinh cosh) / that
            ch, sh2 = torch.cosh(scale * dy), torch.sinh(scale * dy).square()
            den = torch.sin(scale * dx).square() + sh2
            img = torch.sin(scale * sx).square() + sh2
            same = None
            if a == b:
                same = torch.eye(i.stop - a, dtype=torch.bool, device=pos.device)
                den = torch.where(same, math.inf, den)
            pot = torch.log(img) - torch.log(den)
            ex = torch.sin(2 * scale * dx) / den - torch.sin(2 * scale * sx) / img
            ey = 2 * torch.sinh(scale * dy) * ch * (1 / den - 1 / img)
            r2 = dx.square() + dy.square()
            if same is not None:
                r2 = torch.where(same, math.inf, r2)
                pot, ex, ey = (torch.where(same, 0.0, v) for v in (pot, ex, ey))
            close = r2 < (6.0 * soft) ** 2
            soft2 = r2 + soft * soft
            pot = pot - torch.where(close, torch.log(soft2 / r2), 0.0)
            k = torch.where(close, 2 / soft2 - 2 / r2, 0.0)
            phi[i] += pot @ q[j]
            field[0, i] += (scale * ex + k * dx) @ q[j]
            field[1, i] += (scale * ey + k * dy) @ q[j]
    own = torch.sin(2 * scale * pos[0])
    phi += 2 * q * torch.log(own.abs() / scale)
    field[0] -= q * 2 * scale * torch.cos(2 * scale * pos[0]) / own
    return x["k_e"] * phi, x["k_e"] * field


def exact(case: dict, seed: int):
    kind, n = case["kind"], case["n"]
    m = case.get("m", n)
    pairs = float(n) * m * {"sim": 2, "fmm_at": 2, "grad": 1}.get(kind, 1)
    if kind == "strip" or (kind == "grad" and case["loss"] == "field"):
        pairs *= 12
    if pairs > EXACT_PAIRS:
        return None
    x = _inputs(case, seed)
    if kind == "sim":
        return _exact_step(x, case)
    if kind == "strip":
        return _exact_strip(x)
    kernel, eps = case.get("kernel", "log"), _eps(case) if "kernel" in case else 0.0
    if kind in ("direct", "fmm_at", "panels"):
        return _target_sums(x["targets"], x.get("exclude"), x["pos"], x["q"], kernel, eps)
    if kind == "grad" and case["loss"] == "field":
        return _field_loss_gradients(x["pos"], x["q"], x["w"], x["e"], kernel, eps)
    phi, field = _self_sums(x["pos"], x["q"], kernel, eps)
    if kind == "grad":
        return 0.5 * (x["q"] * phi).sum(), -x["q"] * field, phi
    return phi, field
