"""The one-launch solve X = Q U^{-1} L^{-1} P B (getrs) and the refined solve at
the edges of its 64-row blocks and of its groups of right-hand sides, against
the oracle's factors solved in NumPy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 2, 3, 5, 8, 9, 33, 65])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 130, 257, 641])
def test_solve_edges(built, n, nrhs):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(1000 * n + nrhs)
    # diagonally weighted: kappa stays small, so the bound below is the rounding's
    a = rng.standard_normal((n, n)) + 2.0 * np.sqrt(n) * np.eye(n)[rng.permutation(n)]
    b = rng.standard_normal((n, nrhs))
    x = np.linalg.solve(a, b)
    ldb, lda = n + 3, n + 2
    d_a = torch.zeros(n, lda, dtype=torch.float64, device="cuda")
    d_a[:, :n] = torch.from_numpy(a.T.copy()).cuda()
    d_b = torch.full((nrhs, ldb), 7.0, dtype=torch.float64, device="cuda")
    d_b[:, :n] = torch.from_numpy(b.T.copy()).cuda()
    keep = d_b.clone()
    lu = d_a.clone()
    ipiv, jpiv = np.zeros(n, dtype=np.int32), np.zeros(n, dtype=np.int32)
    st, info = dp.getrf_device_ex(n, n, lu, lda, ipiv, jpiv)
    assert st == dp.SUCCESS and info == n
    assert dp.getrs_device(n, nrhs, lu, lda, ipiv, jpiv, d_b, ldb) == dp.SUCCESS
    bound = 1e3 * n * np.finfo(np.float64).eps * max(1.0, np.abs(x).max())
    assert np.abs(d_b[:, :n].cpu().numpy().T - x).max() <= bound
    assert torch.equal(d_b[:, n:], keep[:, n:])  # the padding is not touched
    f = dp.Factor(n, d_a, lda, precision=dp.PRECISION_FP64)
    for policy in (0, 1, -2):  # as many CTAs as fit, one, one per two blocks
        prev = dp.lib().dp_tri_solve_grid(policy)
        try:
            again = keep.clone()
            st, res = f.solve(again, ldb, nrhs)
        finally:
            dp.lib().dp_tri_solve_grid(prev)
        assert st == dp.SUCCESS and res.converged == 1 and res.backward_error <= 1e-14
        assert np.abs(again[:, :n].cpu().numpy().T - x).max() <= bound
        assert torch.equal(again[:, n:], keep[:, n:])
    f.close()


def test_a_nan_right_hand_side_ends(built):
    """Result values wait on their own bit patterns: NaNs of every pattern in B
    (the all-ones pattern that marks a value not yet there among them) must
    come through as NaN, not as a wait that runs out."""
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 200
    a = torch.eye(n, dtype=torch.float64, device="cuda") * 2.0
    ipiv, jpiv = np.zeros(n, dtype=np.int32), np.zeros(n, dtype=np.int32)
    st, info = dp.getrf_device_ex(n, n, a, n, ipiv, jpiv)
    assert st == dp.SUCCESS and info == n
    b = torch.ones(2, n, dtype=torch.float64, device="cuda")
    b.view(torch.int64)[0, 5] = -1
    b.view(torch.int64)[1, 150] = 0x7FF8000000000001
    assert dp.getrs_device(n, 2, a, n, ipiv, jpiv, b, n) == dp.SUCCESS
    got = b.cpu()
    assert bool(torch.isnan(got[0, 5])) and bool(torch.isnan(got[1, 150]))
