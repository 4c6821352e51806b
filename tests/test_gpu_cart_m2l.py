"""The Cartesian M2L with a lane per translation (td3_cart_m2l_rows and, from the moments
themselves, td3_cart_m2l / td3_cart_m2l_mixed) against the oracle's cart_m2l_host on rows
that meet its edges: empty rows, rows of one entry, rows that end on and beside a group's 4
lanes, rows above 256 entries (the whole warp), more rows than a warp's groups, sources up
to 200 times smaller and larger than their destination, zero and positive softening.

Tolerances: FP64 1e-12 of the largest coefficient of the degree.  Mixed: a coefficient times
h_dst^|b| is what it adds to the field of its cell; moments, coefficients and products are
rounded to FP32 (2^-24), relative to the single translations (which cancel in the sum), and
the recurrence and sums of up to p + 300 terms stay within some hundred roundings: 1e-5 of
the cell's largest sum of the translations' magnitudes.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = [0, 1, 3, 4, 5, 0, 8, 31, 32, 33, 255, 256, 257, 300, 0, 64] + [7] * 40 + [0] * 40 + [2] * 7


def _case(order, eps, seed):
    rng = np.random.default_rng(seed)
    counts = np.array(ROWS)
    start = np.concatenate(([0], np.cumsum(counts))).astype(np.int64)
    n_src = 500
    src_half = 0.1 * 2.0 ** rng.integers(-7, 8, n_src)
    dst_half = np.where(np.arange(len(counts)) % 9 == 4, 1e-3, 0.1)
    src_center = rng.uniform(-1, 1, (n_src, 2))
    # every destination outside a circle of four times the largest source cell
    far = 4 * (src_half.max() + 0.1)
    angle = rng.uniform(0, 2 * np.pi, len(counts))
    dst_center = (far + rng.uniform(2, 30, len(counts)))[:, None] * np.stack(
        (np.cos(angle), np.sin(angle)), axis=1)
    partners = rng.integers(0, n_src, start[-1]).astype(np.int64)
    degree = np.array([n for n in range(order + 1) for _ in range(n + 1)])
    moments = rng.normal(size=(n_src, degree.size)) * src_half[:, None] ** degree
    return dict(start=start, partners=partners, dst_center=dst_center, dst_half=dst_half,
                src_center=src_center, src_half=src_half, moments=moments, degree=degree, eps=eps)


def _oracle_locals(oracle, c, order, start=None, dst_center=None):
    t = oracle.cart_tables(order)
    start = c["start"] if start is None else start
    dst_center = c["dst_center"] if dst_center is None else dst_center
    local = np.zeros((start.size - 1, c["degree"].size))
    p = oracle._p
    oracle.lib().cart_m2l_host(p(start), local.shape[0], p(c["partners"]), p(dst_center),
                               p(c["src_center"]), p(c["moments"]), local.shape[1], c["eps"],
                               p(t["ex"]), p(t["ey"]), p(t["rec"]), p(t["m2l"]),
                               p(t["m2l_coef"]), len(t["m2l_coef"]), p(local))
    return local


@pytest.mark.parametrize("order", range(17))
@pytest.mark.parametrize("mixed", [0, 1])
def test_plain_moments_are_scaled_to_the_bits_of_records(order, mixed):
    c = _case(order, 1e-3, 50 + order)
    assert np.array_equal(_run(c, order, mixed, False), _run(c, order, mixed, True))


@pytest.mark.parametrize("order", [4, 12, 16])
@pytest.mark.parametrize("packed", [False, True])
def test_mixed_units_round_nothing(order, packed):
    """The unit of a cell in the mixed form is a power of two: sizes that change within the same
    nearest one, in another ratio to each other, give the same bits."""
    c = _case(order, 1e-3, order)
    want = _run(c, order, 1, packed)
    assert np.isfinite(want).all()
    for scale in (0.93, 1.07):  # 0.1 * 2^k and 1e-3: 1.6 / 16 and 1.024 / 1024, off sqrt(2)
        other = dict(c, src_half=c["src_half"] * scale, dst_half=c["dst_half"] / scale)
        assert np.array_equal(_run(other, order, 1, packed), want)


@pytest.mark.parametrize("size", [1e-28, 1e30])
def test_mixed_charges_near_the_ends_of_fp32(oracle, size):
    """Charges whose moments keep clear of FP32's ends by themselves, but not times the 16th
    power of the largest ratio of a source's size to its destination's, 16 (tolerances above)."""
    order, n = 16, 64
    rng = np.random.default_rng(3)
    degree = np.array([k for k in range(order + 1) for _ in range(k + 1)])
    start = np.arange(n + 1, dtype=np.int64)
    src_half = np.full(n, 0.25)
    dst_half = 0.25 / 2.0 ** (np.arange(n) % 5)
    angle = rng.uniform(0, 2 * np.pi, n)
    c = dict(start=start, partners=np.arange(n, dtype=np.int64), src_half=src_half,
             dst_half=dst_half, src_center=rng.uniform(-1, 1, (n, 2)),
             dst_center=5 * np.stack((np.cos(angle), np.sin(angle)), axis=1), degree=degree,
             moments=size * rng.normal(size=(n, degree.size)) * src_half[:, None] ** degree, eps=0.0)
    want = _oracle_locals(oracle, c, order)
    unit = dst_half[:, None] ** degree
    for packed in (False, True):
        got = _run(c, order, 1, packed)
        error = np.max(np.abs(got - want) * unit, axis=1) / np.max(np.abs(want) * unit, axis=1)
        assert np.all(error < 1e-5)


def _off_by_a_double(t):
    """A copy of ``t`` that starts 8 bytes past a 16-byte boundary."""
    copy = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view_as(t)
    assert copy.data_ptr() % 16 == 8
    return copy.copy_(t)


def _run(c, order, mixed, packed, shift=False):
    from tree_d_3d_b200 import _lib

    d = {k: torch.tensor(v, device="cuda") for k, v in c.items() if isinstance(v, np.ndarray)}
    if shift:
        d = {k: _off_by_a_double(v) for k, v in d.items()}
    n_dst, n_src = c["start"].size - 1, c["src_center"].shape[0]
    local = torch.zeros((n_dst, c["degree"].size), dtype=torch.float64, device="cuda")
    cells = (d["start"].data_ptr(), d["partners"].data_ptr(), n_dst, d["dst_center"].data_ptr(),
             d["dst_half"].data_ptr(), d["src_center"].data_ptr(), d["src_half"].data_ptr())
    if packed:
        width = _lib.lib().td3_cart_record_bytes(order, mixed)
        records = torch.empty(n_src * width, dtype=torch.uint8, device="cuda")
        _lib.call("td3_pack_cart_sources", n_src, order, d["moments"].data_ptr(),
                  d["src_half"].data_ptr(), mixed, records.data_ptr(), _lib.stream())
        _lib.call("td3_cart_m2l_rows", *cells, records.data_ptr(), order, c["eps"], mixed,
                  local.data_ptr(), _lib.stream())
    elif mixed:
        _lib.call("td3_cart_m2l_mixed", *cells, d["moments"].data_ptr(), order, c["eps"],
                  local.data_ptr(), _lib.stream())
    else:
        _lib.call("td3_cart_m2l", *cells[:4], cells[5], d["moments"].data_ptr(), order, c["eps"],
                  0, 0, 0, 0, local.data_ptr(), _lib.stream())
    return local.cpu().numpy()


@pytest.mark.parametrize("order,eps", [(1, 0.0), (4, 1e-3), (5, 0.5), (8, 0.0), (11, 1e-3),
                                       (12, 0.5), (13, 0.5), (14, 0.0), (16, 1e-3)])
def test_cartesian_m2l_rows_match_the_oracle(oracle, order, eps):
    c = _case(order, eps, 100 + order)
    want = _oracle_locals(oracle, c, order)
    filled = np.diff(c["start"]) > 0
    scale = np.array([np.abs(want[:, c["degree"] == n]).max() for n in range(order + 1)])[c["degree"]]
    unit = c["dst_half"][:, None] ** c["degree"]
    # the translations one by one, and the sums of their magnitudes
    row = np.repeat(np.arange(filled.size), np.diff(c["start"]))
    single = _oracle_locals(oracle, c, order, np.arange(row.size + 1, dtype=np.int64),
                            np.ascontiguousarray(c["dst_center"][row]))
    magnitude = np.zeros_like(want)
    np.add.at(magnitude, row, np.abs(single))
    largest = np.max(magnitude * unit, axis=1)

    def error(a, b, mixed):
        if not mixed:
            return np.max(np.abs(a - b) / scale)
        return np.max((np.abs(a - b) * unit).max(1)[filled] / largest[filled])

    for mixed, tol in ((0, 1e-12), (1, 1e-5)):
        packed = _run(c, order, mixed, True)
        assert error(packed, want, mixed) < tol
        assert np.array_equal(packed, _run(c, order, mixed, True))  # the same bits every run
        assert error(_run(c, order, mixed, False), packed, mixed) < tol
        assert not packed[~filled].any()


@pytest.mark.parametrize("order", [3, 12, 16])
@pytest.mark.parametrize("mixed,packed", [(0, False), (0, True), (1, False), (1, True)])
def test_arrays_on_any_double(order, mixed, packed):
    """Rows, partners, centres, sizes and moments that start 8 bytes past a 16-byte boundary."""
    c = _case(order, 1e-3, order)
    assert np.array_equal(_run(c, order, mixed, packed, shift=True), _run(c, order, mixed, packed))


def test_cartesian_records_reject_other_orders():
    from tree_d_3d_b200 import _lib

    lib = _lib.lib()
    assert lib.td3_cart_record_bytes(12, 0) % 16 == 0
    assert lib.td3_cart_record_bytes(17, 0) == _lib.EINVAL
    assert lib.td3_pack_cart_sources(1, 17, 0, 0, 0, 0, 0) == _lib.EINVAL
    assert lib.td3_cart_m2l_rows(0, 0, 1, 0, 0, 0, 0, 0, 17, 0.0, 0, 0, 0) == _lib.EINVAL


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("order", [0, 2, 6, 10, 14])
def test_unpacked_moments_do_not_read_what_shared_memory_held(order, mixed):
    """Orders below their template's: moments above the order count as zero, whatever the
    launch before (NaN moments of the template's order) left in shared memory."""
    c = _case(order, 1e-3, order)
    full = 4 if order <= 4 else 8 if order <= 8 else 12 if order <= 12 else 16
    nans = _case(full, 1e-3, order)
    nans["moments"] = np.full_like(nans["moments"], np.nan)
    for _ in range(5):
        assert np.isnan(_run(nans, full, mixed, True)).any()
        got = _run(c, order, mixed, False)
        assert np.isfinite(got).all()
