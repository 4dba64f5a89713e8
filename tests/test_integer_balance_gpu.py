"""The integer-core trailing update where the rows of U12 are not alike from
column to column: zeros, steps and grading that the columns which set its balance
do not show, at matrix scales from 1e-20 to 1e20.

`_schur` reads one update by itself: the leading 256 x 256 block is a multiple of
I larger than every entry below it, so L21 and U12 are given, and a threshold that
no entry of the Schur complement reaches ends the factorisation after 256 steps.
An FP64 sum of K products is within K u (|L21| |U12|) of the exact one, element by
element; the update has to stay within K + 2 such units."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = np.finfo(np.float64).eps / 2
W = 256
N = 2560
FIRST = 2 * W  # the columns the integer cores take, after the next outer block


def _torch():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _factor(a, **kw):
    import delayed_pivoting as dp

    torch = _torch()
    m, n = a.shape
    d = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    k = min(m, n)
    ipiv, jpiv = np.zeros(k, dtype=np.int32), np.zeros(k, dtype=np.int32)
    st, info = dp.getrf_device_ex(m, n, d, m, ipiv, jpiv, **kw)
    assert st == dp.SUCCESS
    return np.asfortranarray(d.cpu().numpy().T), ipiv, jpiv, info


D = 2.0 ** 62  # the pivots


def _schur(L, R, scale=1.0, **kw):
    """The first update by itself: returns (L21, U12, Schur complement) for
    multipliers L ((N - W) x W, below 0.95) and U12 = scale R (W x (N - W))."""
    a = np.zeros((N, N))
    a[:W, :W] = D * np.eye(W)
    a[W:, :W] = D * L
    a[:W, W:] = R
    f, ip, jp, info = _factor(a * scale, threshold=0.95 * D * scale, **kw)
    assert info == W and np.array_equal(ip, np.arange(N)) and np.array_equal(jp, np.arange(N))
    return f[W:, :W], f[:W, W:], f[W:, W:]


def _operands(seed):
    rng = np.random.default_rng(seed)
    return rng, rng.uniform(-0.9, 0.9, (N - W, W)), 0.05 * rng.standard_normal((W, N - W))


def _exact(L, R, rows):
    return -(L[rows].astype(np.longdouble) @ R.astype(np.longdouble))


# name -> (L, R) made unlike; columns of R count from matrix column W
def _unlike(name, rng, L, R):
    at = FIRST - W
    if name.startswith("step"):  # alternate rows of another size in the columns that come first
        R[1::2, at:at + 64] *= float(name[4:])
    elif name == "zero":  # one row of U12 zero there
        R[7, at:at + 64] = 0.0
    elif name == "late":  # one element far to the right
        R[100, 2000] *= 1e12
    elif name == "graded":  # small rows below, and a step that only they see
        L *= 1e-6
        R[1::2, at:at + 64] *= 1e-6
    elif name == "sparse":
        R *= rng.random(R.shape) < 0.02
    elif name == "arrow":
        R[4:] = 0.0
        L[:, 4:] *= 1e-9
    elif name == "blocks":  # L and U12 meet in few of the steps
        L[:1000, :128] = 0.0
        L[1000:, 128:] = 0.0
        R[:128, 900:] = 0.0
        R[:128, :900] *= 1e-15
    return L, R


@pytest.mark.parametrize("scale", [1.0, 1e-9, 1e9, 1e-20, 1e20])
@pytest.mark.parametrize("name", ["step1e-8", "step1e-20", "step1e8", "step0", "zero", "late",
                                  "graded", "sparse", "arrow", "blocks"])
def test_update_of_unlike_rows(built, name, scale):
    rng, L, R = _operands(3)
    L, R, got = _schur(*_unlike(name, rng, L, R), scale)
    rows = rng.choice(N - W, 160, replace=False)
    err = np.abs(got[rows] - _exact(L, R, rows))
    lim = (W + 2) * U * (np.abs(L[rows]) @ np.abs(R))
    assert (err <= lim).all(), float((err / np.where(lim > 0, lim, np.inf)).max())


@pytest.mark.parametrize("name,scale", [("plain", 1.0), ("plain", 1e-9), ("plain", 1e20),
                                        ("rows", 1.0), ("columns", 1.0), ("zero row", 1e-9),
                                        ("zero column of L", 1e9), ("zero columns", 1e-20)])
def test_like_rows_stay_on_the_integer_cores(built, name, scale):
    """The digits' exact sums are rounded a few times in all: the last additions
    and the subtraction, at most half a unit in the last place of numbers of the
    result's size each, so about 0.6 u of it (root mean square) and 1.5 u with
    room.  An FP64 sum of 256 random products is rounded 256 times: about 3.8 u."""
    rng, L, R = _operands(5)
    if name == "rows":  # small rows of U12 have the large multipliers
        small = 10.0 ** rng.uniform(-6, 0, (W, 1))
        R *= small
        L *= 10.0 ** rng.uniform(-6, 0, (N - W, 1)) / small.T * small.min()
    elif name == "columns":
        R *= 10.0 ** rng.uniform(-40, 0, (1, N - W))
    elif name == "zero row":
        R[7] = 0.0
    elif name == "zero column of L":
        L[:, 9] = 0.0
    elif name == "zero columns":
        R[:, FIRST - W:FIRST - W + 2] = 0.0
        R[:, 1500] = 0.0
    L, R, got = _schur(L, R, scale)
    rows = rng.choice(N - W, 160, replace=False)
    cols = np.arange(FIRST - W, N - W)
    cols = cols[R[:, cols].any(0)]
    want = _exact(L, R[:, cols], rows)
    assert not got[:, (R == 0.0).all(0)].any()
    # each element in units of its row's and column's size
    ms = (want / want.astype(np.float64).std()).astype(np.float64) ** 2
    size = np.sqrt(ms.mean(1, keepdims=True) * ms.mean(0, keepdims=True) / ms.mean())
    rel = ((got[rows][:, cols] - want) / want.astype(np.float64).std()).astype(np.float64) / size
    assert np.sqrt((rel ** 2).mean()) <= 1.5 * U


@pytest.mark.parametrize("scale,row", [(1e-9, 0.0), (1e9, 0.0), (1e-20, 0.0), (1.0, 1e-12)])
def test_factors_of_unlike_columns(built, scale, row):
    """Columns 512 .. 575 sparse beside a full diagonal, the first pivot row zero
    in them; or the first pivot row small in them only."""
    import oracle as orc

    _torch()
    rng = np.random.default_rng(17)
    a = rng.standard_normal((N, N))
    s = slice(512, 576)
    if row == 0.0:
        a[:, s] *= rng.random((N, 64)) < 0.02
        a[np.arange(512, 576), np.arange(512, 576)] += 1.0
    a[np.abs(a[:, 0]).argmax(), s] *= row
    a = np.asfortranarray(a * scale)
    f, ip, jp, info = _factor(a)
    ri, rj, rinfo = orc.oracle_getrf(a.copy(order="F"))
    assert info == rinfo == N
    np.testing.assert_array_equal(ip, ri)
    np.testing.assert_array_equal(jp, rj)
    p = np.arange(N)
    for k in range(N):
        p[[k, ip[k]]] = p[[ip[k], k]]
    lower, upper = np.tril(f, -1) + np.eye(N), np.triu(f)
    err = np.abs(a[p] - lower @ upper)  # (the check's own product adds as much again)
    assert (err <= 2 * N * U * (np.abs(lower) @ np.abs(upper))).all()


def test_schedules_agree_when_a_later_part_is_unlike(built):
    """The first 256 columns of the integer update are alike, the ones after them
    not: both schedules hand the same columns back to the FP64 kernel."""
    rng, L, R = _operands(11)
    R[np.arange(W) % 8 != 0, 2 * W:] *= 1e-15
    on, off = _schur(L, R, lookahead=1)[2], _schur(L, R, lookahead=2)[2]
    np.testing.assert_array_equal(on, off)
