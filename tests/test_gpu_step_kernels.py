"""The simulation step's own kernels against the same step on array operations: sizes around
a warp and a block, with and without a magnetic field, fixed and uncharged particles, walls
that absorb some.  Both forms do the same operations in FP64 (sines by another routine), so
1e-13 of the largest value.  Each step is compared on the native step's own state and fields:
the fields of a tree are not continuous in the positions (a particle changes its cell).
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import relative

pytestmark = pytest.mark.gpu


def _simulation(n, b_z, kind):
    from tree_d_3d_b200 import Quad
    from tree_d_3d_b200.simulation import ElectrostaticSimulation

    rng = np.random.default_rng(n)
    charges, fixed = rng.choice([-1.0, 1.0], n), np.zeros(n, dtype=bool)
    if kind == "mixed":
        charges[::3] = 0.0
        fixed[1::4] = True
    return ElectrostaticSimulation(
        positions=rng.uniform(-0.9, 0.9, (2, n)), velocities=rng.normal(size=(2, n)),
        charges=charges, masses=rng.uniform(0.5, 2, n), fixed=fixed, bounds=Quad(0, 0, 1),
        k_e=1e-2, softening=1e-2, dt=0.05, B_z=b_z, kernel="log" if kind == "log" else "coulomb",
        absorbing_walls={"x_max": 0.95, "y_min": -0.95} if kind != "free" else {"x_min": -50.0})


@pytest.mark.parametrize("n", [1, 2, 31, 33, 257, 1500])
@pytest.mark.parametrize("b_z,kind", [(0.0, "free"), (1.5, "free"), (1.5, "mixed"), (0.7, "log")])
def test_native_step_matches_the_array_step(n, b_z, kind):
    from tree_d_3d_b200.simulation import ElectrostaticSimulation

    from tree_d_3d_b200.simulation import _drift

    sim = _simulation(n, b_z, kind)
    assert sim._native()
    for _ in range(3):
        sim.compute_fields(include_fixed=False, potential=False)
        pos, vel, electric = sim.positions, sim.velocities, sim._electric
        q, m, mobile = sim.charges, sim.masses, (~sim.fixed).double()
        sim.step()
        vel = vel + 0.5 * sim.dt * electric / m * mobile
        pos, vel = _drift(pos, vel, q, m, sim.B_z, sim.dt, mobile)
        inside = torch.ones_like(q, dtype=torch.bool)
        for _, axis, sign, value in sim._walls:
            inside &= ~(sign * (pos[axis] - value) > 0)
        assert sim.num_particles == int(inside.sum())
        if not sim.num_particles:
            break
        pos, vel, q, m, mobile = pos[:, inside], vel[:, inside], q[inside], m[inside], mobile[inside]
        vel = vel + 0.5 * sim.dt * sim._electric / m * mobile
        forces = sim._electric + q * sim.B_z * torch.stack((vel[1], -vel[0]))
        for a, b in ((sim.positions, pos), (sim.velocities, vel), (sim.forces, forces)):
            assert relative(a.cpu().numpy(), b.cpu().numpy()) < 1e-13


def test_step_sees_a_state_changed_in_place_and_refuses_non_finite_positions():
    sim = _simulation(100, 1.0, "free")
    sim.compute_fields()
    before = sim._electric.clone()
    sim.compute_fields()
    assert torch.equal(sim._electric, before)
    sim.charges[3] *= 2
    sim.compute_fields()
    assert not torch.equal(sim._electric, before)
    sim.positions[0, 5] = float("nan")
    with pytest.raises(ValueError, match="finite"):
        sim.step()


def test_fields_of_a_transposed_state_are_not_taken_for_another_of_the_same_memory():
    """The saved state is compared by its values: positions given as a.T and then, of the same
    numbers in memory, as a.reshape(2, n) are two states."""
    from tree_d_3d_b200 import Quad
    from tree_d_3d_b200.simulation import ElectrostaticSimulation

    n = 500
    rng = np.random.default_rng(7)
    a = torch.tensor(rng.uniform(-0.9, 0.9, (n, 2)), device="cuda")

    def simulation(positions):
        return ElectrostaticSimulation(positions=positions, charges=np.ones(n), bounds=Quad(0, 0, 1),
                                       k_e=1e-2, softening=1e-2, method="fmm")

    sim = simulation(a.T)
    for positions in (a.T, a.reshape(2, n), a.T):
        sim.positions = positions
        sim.compute_fields()
        want = simulation(positions.clone(memory_format=torch.contiguous_format))
        want.compute_fields()
        assert relative(sim._electric.cpu().numpy(), want._electric.cpu().numpy()) < 1e-13
    # a saved state of other strides (of an object kept from elsewhere) is compared as arrays
    pos, *rest = sim._field_state
    sim._field_state = (a.T, *rest)
    sim.positions = a.reshape(2, n)
    assert sim._native() and sim._scan() is None and not sim._fields_current()


@pytest.mark.parametrize("kernel", ["coulomb", "log"])
def test_direct_sums_of_a_strided_state(kernel):
    """Direct fields and the exact pair energy of positions that are a transposed array and
    charges that are every second one of an array."""
    from tree_d_3d_b200 import Quad
    from tree_d_3d_b200.simulation import ElectrostaticSimulation

    n = 500
    rng = np.random.default_rng(8)
    a = torch.tensor(rng.uniform(-0.9, 0.9, (n, 2)), device="cuda")
    q = torch.tensor(rng.normal(size=2 * n), device="cuda")[::2]
    sims = [ElectrostaticSimulation(positions=a.T, charges=q, bounds=Quad(0, 0, 1), k_e=1e-2,
                                    softening=1e-2, kernel=kernel) for _ in range(2)]
    sims[0].positions, sims[0].charges = a.T, q
    for include_fixed in (True, False):
        for sim in sims:
            sim._field_state = None
            sim.compute_fields(include_fixed=include_fixed)
        assert relative(sims[0]._electric.cpu().numpy(), sims[1]._electric.cpu().numpy()) < 1e-13
    energy = [sim.get_potential_energy(exact=True) for sim in sims]
    assert abs(energy[0] - energy[1]) <= 1e-12 * abs(energy[1])


def test_velocities_that_autograd_follows_step_on_array_operations():
    sim = _simulation(50, 1.0, "free")
    sim.velocities.requires_grad_(True)
    assert not sim._native()
    v = sim.velocities
    sim.step()
    sim.velocities.sum().backward()
    assert v.grad is not None


def test_forward_mode_tangents_of_a_step():
    """Tangents of the velocities go through the array operations: with no charge and no
    field a step moves by dt v."""
    from torch.autograd import forward_ad

    sim = _simulation(40, 0.0, "free")
    sim.k_e = 0.0
    tangent = torch.randn_like(sim.velocities)
    with forward_ad.dual_level():
        sim.velocities = forward_ad.make_dual(sim.velocities, tangent)
        assert not sim._native()
        sim.step()
        moved = forward_ad.unpack_dual(sim.positions).tangent
        assert torch.allclose(moved, sim.dt * tangent, rtol=1e-14, atol=0)
    assert sim.velocities.is_cuda


def test_step_under_torch_func_jvp():
    sim = _simulation(40, 0.0, "free")
    sim.k_e = 0.0
    start, tangent = sim.velocities.clone(), torch.randn_like(sim.velocities)

    def positions(velocities):
        sim.velocities = velocities
        sim.step()
        return sim.positions

    _, moved = torch.func.jvp(positions, (start,), (tangent,))
    assert torch.allclose(moved, sim.dt * tangent, rtol=1e-14, atol=0)


@pytest.mark.parametrize("shape", [(), (60,)])
def test_magnetic_field_as_a_tensor(shape):
    """B_z as a scalar or per-particle tensor: the array step, with gradients to it."""
    sims = [_simulation(60, 1.25, "free") for _ in range(2)]
    b_z = torch.full(shape, 1.25, dtype=torch.float64, device="cuda", requires_grad=True)
    sims[1].B_z = b_z
    assert sims[0]._native() and not sims[1]._native()
    for sim in sims:
        sim.step()
    assert relative(sims[1].positions.detach().cpu().numpy(),
                    sims[0].positions.cpu().numpy()) < 1e-13
    assert relative(sims[1].velocities.detach().cpu().numpy(),
                    sims[0].velocities.cpu().numpy()) < 1e-11
    (grad,) = torch.autograd.grad(sims[1].positions.sum(), b_z)
    assert grad.shape == b_z.shape and bool(grad.abs().sum() > 0)


@pytest.mark.parametrize("how", ["subclass", "instance"])
def test_step_calls_an_overridden_compute_fields(how):
    """A program's own compute_fields (here: a uniform force added to the charges') gives both
    half kicks of a step."""
    from tree_d_3d_b200.simulation import ElectrostaticSimulation

    class Tilted(ElectrostaticSimulation):
        def compute_fields(self, include_fixed=True, potential=True):
            self._field_state = None
            tree = super().compute_fields(include_fixed, potential)
            self._electric = self._electric + 3.0
            return tree

    sim = _simulation(30, 0.0, "free")
    sim.k_e = 0.0
    if how == "subclass":
        sim.__class__ = Tilted
    else:
        def fields(include_fixed=True, potential=True):
            sim._electric = torch.full_like(sim.positions, 3.0)

        sim.compute_fields = fields
    before = sim.velocities
    sim.step()
    assert torch.allclose(sim.velocities, before + sim.dt * 3.0 / sim.masses, rtol=1e-13, atol=1e-14)
    assert torch.equal(sim.forces, torch.full_like(sim.forces, 3.0))


def test_pair_sum_logarithm_and_reciprocal():
    """direct_field of the log kernel at single distances: phi = -ln r^2 and E = 2 / r to a few
    units in the last place at every magnitude (the table's intervals, both sides of r = 1,
    where ln r^2 must keep its relative accuracy, and beyond the short form's range)."""
    from tree_d_3d_b200 import direct_field

    rng = np.random.default_rng(0)
    near = 1 + np.concatenate([s * 2.0 ** -np.arange(1.0, 50.0) for s in (1, -1)])
    r = np.concatenate([np.exp(rng.uniform(-300, 300, 20000)), rng.uniform(0.5, 2, 20000), near,
                        2.0 ** np.arange(-530, 505.0), [1.0, 1e-155, 1e-160, 1e153, 1e154]])
    phi, field = direct_field(torch.tensor(np.stack((r, 0 * r)), device="cuda"),
                              torch.zeros((2, 1), device="cuda", dtype=torch.float64),
                              torch.ones(1, device="cuda", dtype=torch.float64), kernel="log")
    r2 = r * r
    with np.errstate(over="ignore"):
        want, inverse = -np.log(r2), 2 / r2 * r
    assert not field[1].cpu().numpy()[np.isfinite(inverse)].any()
    for got, ref in ((phi.cpu().numpy(), want), (field[0].cpu().numpy(), inverse)):
        finite = np.isfinite(ref)  # 2 / r^2 of a denormal r^2 is infinite
        assert np.array_equal(got[~finite], ref[~finite])
        assert np.all(np.abs(got[finite] - ref[finite]) <= 4 * np.spacing(np.abs(ref[finite])))


@pytest.mark.parametrize("sources", [1, 2, 3])
def test_pair_sum_reciprocal_root(sources):
    """direct_field of the Coulomb kernel at single distances: phi = 1 / r and E = 1 / r^2 over
    all magnitudes, past the largest and smallest normal r^2, beside sources without charge (the
    pairs are summed two at a time).  Units in the last place: 1 for the root of the rounded
    r^2 (half of r^2's half, and the function's 1 at most), E three of those and three products."""
    from tree_d_3d_b200 import direct_field

    rng = np.random.default_rng(1)
    near = 1 + np.concatenate([s * 2.0 ** -np.arange(1.0, 50.0) for s in (1, -1)])
    r = np.concatenate([np.exp(rng.uniform(-300, 300, 20000)), rng.uniform(0.5, 2, 20000), near,
                        2.0 ** np.arange(-530, 505.0), [1.0, 1e-155, 1e-160, 1e153, 1e154, 1e160]])
    source = np.zeros((2, sources))
    charge = np.zeros(sources)
    charge[sources // 2] = 1.0
    phi, field = direct_field(torch.tensor(np.stack((r, 0 * r)), device="cuda"),
                              torch.tensor(source, device="cuda"),
                              torch.tensor(charge, device="cuda"))
    with np.errstate(over="ignore"):
        r2 = r * r
        want = 1 / np.sqrt(r2.astype(np.longdouble))
        cube = (want.astype(np.float64) ** 3).astype(np.longdouble) * r
    for got, ref, units in ((phi, want, 2), (field[0], cube, 8)):
        got, ref = got.cpu().numpy(), ref.astype(np.float64)
        normal = np.isfinite(ref) & (ref >= 2.0 ** -1000)
        if units == 8:  # 1 / r^3 is normal, too
            normal &= (r < 1e102) & (r > 1e-102)
        assert np.all(np.abs(got[normal] - ref[normal]) <= units * np.spacing(ref[normal]))
        assert not np.isnan(got[r2 > 0]).any()
    big = np.isinf(r2)
    assert big.any() and not phi.cpu().numpy()[big].any()


@pytest.mark.parametrize("call", ["direct", "walk", "fmm"])
def test_log_pairs_beyond_the_reciprocals_range(call):
    """E = 2 q d / r^2 of line charges whose 1 / r^2 alone would overflow, or be denormal."""
    from tree_d_3d_b200 import FlatQuadtree, Quad, direct_field

    for r, q in ((1e-157, 1e-200), (3e-156, 1e-180), (1e-100, 1e-250), (1e153, 1e200), (7e153, 1e250)):
        pos = np.array([[0.0, r], [0.0, 0.0]])
        charge = np.full(2, q)
        if call == "direct":
            phi, field = direct_field(pos, pos, charge, exclude=np.arange(2), kernel="log")
        else:
            tree = FlatQuadtree(pos, charge, Quad(0, 0, 4 * r), kernel="log", order=2)
            phi, field = (tree.fmm() if call == "fmm" else
                          tree.evaluate(pos, exclude=np.arange(2)))
        r2 = r * r  # denormal for the first two
        want = 2 * q / r2 * r
        assert np.isfinite(want) and abs(want) > 0
        assert np.all(np.abs(field[0] - [-want, want]) <= 8 * np.spacing(want)), (r, q)
        assert np.all(np.abs(phi + q * np.log(r2)) <= 8 * np.spacing(abs(q * np.log(r2))))
