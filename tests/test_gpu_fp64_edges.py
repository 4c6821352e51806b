"""The FP64 pair loops and the traversal where their splits change: chunks and odd source
counts of the direct sum, opening tests that hold with equality, generations of less than a
tile to many tiles, and lists that outgrow their first buffers.

The sums agree with the oracle's to 1e-12 normwise (at most 3000 terms of a few ulp each, in
another order); lists are whole numbers and equal.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import relative

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("kernel", ["coulomb", "log"])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 129, 257])
def test_direct_sum_chunk_edges(oracle, kernel, n):
    from tree_d_3d_b200 import direct_field

    rng = np.random.default_rng(n)
    pos = rng.uniform(-1, 1, (2, n))
    q = rng.normal(size=n)
    q[n // 2] = 0.0
    for targets, exclude in ((pos, np.arange(n)), (rng.uniform(-1, 1, (2, 131)), None)):
        ref = oracle.direct_field(targets, pos, q, exclude=exclude, kernel=kernel)
        got = direct_field(targets, pos, q, exclude=exclude, kernel=kernel)
        assert relative(got[0], ref[0]) < TOL and relative(got[1], ref[1]) < TOL


@pytest.mark.parametrize("theta", [-0.5, 0.0, 0.25, 0.5, 1.0])
@pytest.mark.parametrize("leaf", [1, 3, 8])
def test_walk_opens_cells_at_equality(oracle, theta, leaf):
    """Targets on a dyadic grid around dyadic cells: |r| = 2 h / theta exactly for many of
    them, where the cell is opened; so is every cell for theta <= 0."""
    from tree_d_3d_b200 import FlatQuadtree, Quad

    rng = np.random.default_rng(leaf)
    pos, q = rng.uniform(-1, 1, (2, 3000)), rng.choice([-1.0, 1.0], 3000)
    side = (np.arange(32) - 15.5) / 16
    targets = np.stack([a.ravel() for a in np.meshgrid(side, side)])
    ref = oracle.OracleTree(pos, q, (0, 0, 1), leaf_capacity=leaf).evaluate(
        targets, theta=theta, softening=1e-3)
    got = FlatQuadtree(pos, q, Quad(0, 0, 1), leaf_capacity=leaf).evaluate(
        targets, theta=theta, softening=1e-3)
    assert relative(got[0], ref[0]) < TOL and relative(got[1], ref[1]) < TOL


@pytest.mark.parametrize("n", [1, 9, 400, 1500, 6000])
@pytest.mark.parametrize("theta", [0.05, 0.5, 0.9])
def test_traversal_lists_from_part_of_a_tile_to_many(oracle, n, theta):
    from tree_d_3d_b200 import FlatQuadtree, Quad

    rng = np.random.default_rng(n)
    pos, q = rng.uniform(-1, 1, (2, n)), np.ones(n)
    m2l, p2p = oracle.OracleTree(pos, q, (0, 0, 1), kernel="log", order=4).lists(theta)
    lists = FlatQuadtree(pos, q, Quad(0, 0, 1), kernel="log", order=4)._lists(theta)
    assert np.array_equal(lists["m2l"].cpu().numpy(), m2l)
    assert np.array_equal(lists["p2p"].cpu().numpy(), p2p)
