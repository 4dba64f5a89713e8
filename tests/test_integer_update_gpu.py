"""The trailing update on the integer tensor cores, inside factorisations large
enough to use it: records and residuals against the oracle for N(0, 1) entries,
delays, rows and columns of very different size, ragged shapes, and operands it
hands back to the FP64 kernel (NaN, infinities, extreme scales); and both
schedules bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(dp, torch, a, lookahead=0, nb_outer=0):
    m, n = a.shape
    d = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    k = min(m, n)
    ipiv, jpiv = np.zeros(k, dtype=np.int32), np.zeros(k, dtype=np.int32)
    st, info = dp.getrf_device_ex(m, n, d, m, ipiv, jpiv, lookahead=lookahead, nb_outer=nb_outer)
    assert st == dp.SUCCESS
    return np.asfortranarray(d.cpu().numpy().T), ipiv, jpiv, info, dp.getrf_last_report()


def _matrix(kind, m, n):
    rng = np.random.default_rng(m * 7 + n)
    a = rng.standard_normal((m, n))
    if kind == "delays":
        a[:, rng.choice(n, 6, replace=False)] = 0.0
        a[:, rng.choice(n, 6, replace=False)] *= 1e-18
    elif kind == "rows":
        a *= 10.0 ** rng.uniform(-6, 6, (m, 1))
    elif kind == "columns":
        a *= 10.0 ** rng.uniform(-40, 40, (1, n))
    elif kind == "extreme":
        a[:, -1] *= 1e200  # beyond the scales the digits cover
    return np.asfortranarray(a)


@pytest.mark.parametrize("kind,m,n,nb_outer", [
    ("plain", 2900, 2900, 0), ("delays", 3001, 2877, 0), ("rows", 2800, 2800, 0),
    ("columns", 2800, 2800, 0), ("extreme", 2800, 2800, 0), ("plain", 4000, 2300, 128),
    ("plain", 2000, 3900, 200)])
def test_records_and_residual(built, kind, m, n, nb_outer):
    import delayed_pivoting as dp
    import oracle as orc
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    a = _matrix(kind, m, n)
    f, ip, jp, info, report = _run(dp, torch, a, nb_outer=nb_outer)
    ri, rj, rinfo = orc.oracle_getrf(a.copy(order="F"))
    assert report["near_ties"] == 0 and info == rinfo
    np.testing.assert_array_equal(ip, ri)
    np.testing.assert_array_equal(jp, rj)
    scale = np.abs(a).max(axis=1, keepdims=True) if kind == "rows" else np.ones((m, 1))
    cols = np.abs(a).max(axis=0, keepdims=True) if kind in ("columns", "extreme", "delays") else np.ones((1, n))
    cols[cols == 0.0] = 1.0
    # row by row and column by column: P A Q - L U in units of each row's and column's size
    p, q = np.arange(m), np.arange(n)
    for k in range(info):
        p[[k, ip[k]]] = p[[ip[k], k]]
        q[[k, jp[k]]] = q[[jp[k], k]]
    L = np.tril(f[:, :info], -1)
    L[np.arange(info), np.arange(info)] = 1.0
    r = (a[p][:, q] - L @ np.triu(f[:info])) / scale[p] / cols[:, q]
    r[info:, info:] = 0.0
    unit = np.finfo(np.float64).eps / 2
    assert np.linalg.norm(r) <= 10.0 * unit * max(m, n) * np.linalg.norm(a / scale / cols)


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_non_finite_operands_take_the_fp64_kernel(built, value):
    import delayed_pivoting as dp
    import oracle as orc
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    a = _matrix("plain", 2800, 2800)
    a[1700, 2750] = value  # in the trailing part of every block before its own
    f, ip, jp, info, _ = _run(dp, torch, a)
    ref = a.copy(order="F")
    ri, rj, rinfo = orc.oracle_getrf(ref)
    k = 2700  # up to the columns the value reaches the records agree, and it stays in its column
    assert info == rinfo
    np.testing.assert_array_equal(ip[:k], ri[:k])
    np.testing.assert_array_equal(np.isfinite(f[:, :k]), np.isfinite(ref[:, :k]))
    np.testing.assert_array_equal(np.isnan(f[:, 2750]), np.isnan(ref[:, 2750]))


def test_both_schedules_bit_for_bit(built):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    a = _matrix("delays", 3300, 3300)
    f1, i1, j1, info1, _ = _run(dp, torch, a, lookahead=1)
    f2, i2, j2, info2, _ = _run(dp, torch, a, lookahead=2)
    assert info1 == info2
    np.testing.assert_array_equal(i1, i2)
    np.testing.assert_array_equal(j1, j2)
    np.testing.assert_array_equal(f1, f2)
