"""The Cartesian moments and L2L of orders up to 16 (their own kernels) at the edges of their
templates, on trees with empty cells, leaves of many particles and levels of one node.

The moments of a degree do not depend on the order, so those of order 20 (a block per node)
must hold the same bits; the L2L shifts in another order of operations than the oracle's rows
and must agree within 1e-12 of the largest coefficient of a degree.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
ORDERS = [(1, 3), (4, 8), (5, 40), (8, 8), (9, 100), (12, 8), (13, 33), (16, 8)]


def _points(seed):
    rng = np.random.default_rng(seed)
    return np.concatenate([rng.uniform(-1, 1, (2, 3000)), rng.normal(0.3, 0.003, (2, 2000))], 1), rng


def _tree(pos, q, order, capacity):
    from tree_d_3d_b200 import FlatQuadtree, Quad

    return FlatQuadtree(torch.tensor(pos, device="cuda"), torch.tensor(q, device="cuda"),
                        Quad(0, 0, 1), order=order, leaf_capacity=capacity)


def _adjoint_moments(tree, w, e):
    from tree_d_3d_b200 import _cartesian, _lib

    t = tree._cartesian_tables()
    out = torch.empty((tree.node_count, _cartesian.size(tree.order)), dtype=torch.float64,
                      device="cuda")
    levels = np.ascontiguousarray(tree.levels, dtype=np.int64)
    _lib.call("td3_cart_moments_adjoint", levels.ctypes.data, len(levels) - 1,
              tree._sorted_pos.data_ptr(), w.data_ptr(), e.data_ptr(), tree.pos.shape[1],
              tree.node_center.data_ptr(), tree.node_start.data_ptr(), tree.node_end.data_ptr(),
              tree.node_child.data_ptr(), t["ex"].data_ptr(), t["ey"].data_ptr(),
              t["shift"].data_ptr(), t["shift_coef"].data_ptr(), t["shift_start"].data_ptr(),
              out.shape[1], out.data_ptr(), _lib.stream())
    return out


@pytest.mark.parametrize("order,capacity", ORDERS)
def test_cartesian_moments_equal_those_of_a_higher_order(order, capacity):
    pos, rng = _points(order + capacity)
    q = rng.normal(size=pos.shape[1])
    w, e = torch.tensor(rng.normal(size=q.size), device="cuda"), \
        torch.tensor(rng.normal(size=(2, q.size)), device="cuda")
    low, high = _tree(pos, q, order, capacity), _tree(pos, q, 20, capacity)
    n = (order + 1) * (order + 2) // 2
    assert torch.equal(low._cartesian_moments(), high._cartesian_moments()[:, :n])
    assert torch.equal(_adjoint_moments(low, w, e), _adjoint_moments(high, w, e)[:, :n])


@pytest.mark.parametrize("order,capacity", ORDERS)
def test_cartesian_l2l_matches_the_oracle(oracle, order, capacity):
    pos, rng = _points(7 * order + capacity)
    tree = _tree(pos, np.ones(pos.shape[1]), order, capacity)
    degree = np.array([n for n in range(order + 1) for _ in range(n + 1)])
    # a cell's coefficients of degree n are of the size of its half-width to the -n
    local = rng.normal(size=(tree.node_count, degree.size)) * \
        tree.node_half.cpu().numpy()[:, None] ** -degree
    got = torch.tensor(local, device="cuda")
    tree._cart_downward(tree, got)
    got, want = got.cpu().numpy(), local.copy()
    t, p = oracle.cart_tables(order), oracle._p
    levels = np.ascontiguousarray(tree.levels, dtype=np.int64)
    oracle.lib().cart_downward(p(levels), len(levels), p(tree.node_center.cpu().numpy()),
                               p(tree.node_child.cpu().numpy()), p(t["mono_parent"]),
                               p(t["mono_dir"]), p(t["shift"]), p(t["shift_coef"]),
                               len(t["shift_coef"]), p(want), want.shape[1])
    for level in range(len(levels) - 1):
        rows = slice(levels[level], levels[level + 1])
        for n in range(order + 1):
            a, b = got[rows][:, degree == n], want[rows][:, degree == n]
            assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))


@pytest.mark.parametrize("order,capacity", [(16, 1), (31, 8), (32, 9), (33, 40), (63, 7), (64, 17)])
def test_log_moments_of_high_orders_equal_the_oracle(oracle, order, capacity):
    """Orders above 15 (a warp per node, 8 particles at a time): the oracle's bits."""
    from tree_d_3d_b200 import FlatQuadtree, Quad

    rng = np.random.default_rng(order)
    pos = np.concatenate([rng.uniform(-1, 1, (2, 500)), rng.normal(0.3, 0.01, (2, 500))], 1)
    q = rng.normal(size=1000)
    ref = oracle.OracleTree(pos, q, (0, 0, 1), kernel="log", order=order, leaf_capacity=capacity)
    tree = FlatQuadtree(pos, q, Quad(0, 0, 1), kernel="log", order=order, leaf_capacity=capacity)
    for name in ("node_qabs", "moment_re", "moment_im"):
        got = getattr(tree, name)
        np.testing.assert_array_equal(got.cpu().numpy(), getattr(ref, name))
