"""The FP64 log M2L with a lane per translation (orders up to 20, td3_fmm_m2l) against the
oracle's fmm_m2l_host at the edges of its templates and of its walk over the rows: empty
rows, rows of one entry, on and beside a group's 4 lanes, above the whole-warp lengths, few
rows and many; to 1e-12 of the largest coefficient of a degree, the same bits every run.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = [0, 1, 3, 4, 5, 0, 8, 9, 31, 32, 33, 255, 256, 257, 300, 0, 64] + [7] * 40 + [0] * 40


@pytest.mark.parametrize("order,copies", [(1, 1), (4, 300), (5, 1), (8, 300), (10, 1), (11, 1),
                                          (12, 300), (13, 1), (16, 1), (17, 1), (18, 1), (20, 300)])
def test_log_m2l_rows_match_the_oracle(oracle, order, copies):
    from tree_d_3d_b200 import _lib
    from tree_d_3d_b200.flat_tree import _m2l_coefficients

    rng = np.random.default_rng(order)
    counts = np.array(ROWS * copies)
    n_dst, n_src, w = counts.size, 400, order + 1
    start = np.concatenate(([0], np.cumsum(counts))).astype(np.int64)
    partners = rng.integers(0, n_src, start[-1]).astype(np.int64)
    src = rng.uniform(-1, 1, (n_src, 2))
    angle = rng.uniform(0, 2 * np.pi, n_dst)
    dst = rng.uniform(4, 8, n_dst)[:, None] * np.stack((np.cos(angle), np.sin(angle)), axis=1)
    mre, mim = rng.normal(size=(n_src, w)), rng.normal(size=(n_src, w))
    mim[:, 0] = 0.0  # the charges are real
    coeff = _m2l_coefficients(order, False)
    want_re, want_im = np.zeros((n_dst, w)), np.zeros((n_dst, w))
    p = oracle._p
    oracle.lib().fmm_m2l_host(p(start), n_dst, p(partners), p(dst), p(src), p(mre), p(mim),
                              p(np.ascontiguousarray(coeff)), p(want_re), p(want_im), order)
    d = [torch.tensor(a, device="cuda") for a in (start, partners, dst, src, mre, mim, coeff)]
    runs = []
    for again in range(2):
        if again:  # every array on an odd double: 8 bytes past a 16-byte boundary
            d = [torch.cat((t.reshape(-1)[:1], t.reshape(-1)))[1:] for t in d]
            assert all(t.data_ptr() % 16 == 8 for t in d)
        re = torch.zeros((n_dst, w), dtype=torch.float64, device="cuda")
        im = torch.zeros_like(re)
        _lib.call("td3_fmm_m2l", d[0].data_ptr(), d[1].data_ptr(), n_dst, d[2].data_ptr(),
                  d[3].data_ptr(), d[4].data_ptr(), d[5].data_ptr(), order, d[6].data_ptr(),
                  re.data_ptr(), im.data_ptr(), _lib.stream())
        runs.append((re, im))
    assert torch.equal(runs[0][0], runs[1][0]) and torch.equal(runs[0][1], runs[1][1])
    for got, want in ((runs[0][0], want_re), (runs[0][1], want_im)):
        got = got.cpu().numpy()
        if want is want_im:  # Im b_0 never enters the field (its branch is not fixed)
            got, want = got[:, 1:], want[:, 1:]
        assert np.all(np.max(np.abs(got - want), 0) <= 1e-12 * np.max(np.abs(want), 0))


@pytest.mark.parametrize("order", [5, 9, 11])
def test_powers_above_the_order_may_overflow(order):
    """Cells so small that 1 / t^k overflows above the order only: lengths of 2^-k and the
    field of 2^k are exact, so the scaled solve agrees to the rounding of its logarithms."""
    from tree_d_3d_b200 import FlatQuadtree, Quad

    rng = np.random.default_rng(order)
    pos, q = rng.uniform(-1, 1, (2, 4000)), rng.normal(size=4000)
    scale = 2.0 ** -{5: 133, 9: 96, 11: 82}[order]
    _, want = FlatQuadtree(pos, q, Quad(0, 0, 1), kernel="log", order=order).fmm()
    _, got = FlatQuadtree(scale * pos, q, Quad(0, 0, scale), kernel="log", order=order).fmm()
    assert np.isfinite(got).all()
    assert np.max(np.abs(got * scale - want)) < 1e-12 * np.max(np.abs(want))
