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


def test_traversal_whose_waits_run_out_returns_an_error():
    """No polls: the second tile of a generation gives up waiting for the first.  The call ends
    with an error, also with many tiles and blocks, and the next one gives the lists."""
    import torch

    from tree_d_3d_b200 import FlatQuadtree, Quad, _lib

    lib = _lib.lib()
    rng = np.random.default_rng(4)
    for n, theta in ((40, 0.5), (3000, 0.5), (30_000, 0.3)):
        tree = FlatQuadtree(rng.uniform(-1, 1, (2, n)), np.ones(n), Quad(0, 0, 1), kernel="log",
                            order=4)
        want = tree._lists(theta)
        capacity = [int(want[k].shape[0]) + 1 for k in ("m2l", "p2p")] + [3_000_000]
        lists = [torch.zeros((c, 2), dtype=torch.int64, device="cuda") for c in capacity[:2]]
        ws = _lib.workspace(lib.td3_fmm_traverse_workspace_size(capacity[2], tree.node_count),
                            tree.device)
        sizes = np.zeros(4, dtype=np.int64)

        def traverse(polls):
            return lib.td3_fmm_traverse_polls(
                tree.node_center.data_ptr(), tree.node_half.data_ptr(), tree.node_start.data_ptr(),
                tree.node_end.data_ptr(), tree.node_child.data_ptr(), tree.node_count, theta,
                lists[0].data_ptr(), capacity[0], lists[1].data_ptr(), capacity[1], capacity[2],
                sizes.ctypes.data, polls, ws.data_ptr(), ws.numel(), _lib.stream())

        for _ in range(3):
            rc = traverse(0)
            assert rc == (_lib.OK if n == 40 else _lib.ECUDA)
            assert n == 40 or b"bounded wait" in lib.td3_last_error()
        assert traverse(1 << 22) == _lib.OK
        for got, name, size in zip(lists, ("m2l", "p2p"), sizes):
            assert size == want[name].shape[0] and torch.equal(got[:size], want[name])
        assert traverse(-1) == traverse((1 << 22) + 1) == _lib.EINVAL
