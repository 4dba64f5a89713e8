"""The residual of a solve, by its kernel and by the update kernel: at the edge
between the two (16 right-hand sides, n nrhs = 2^17), padded and ragged, the
reported backward error is that of the returned X to the residual's rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0**-53


@pytest.mark.parametrize("n,nrhs", [(2047, 64), (2048, 64), (1261, 104), (1260, 104), (4099, 32), (700, 15),
                                    (1111, 130)])
def test_reported_error(n, nrhs):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator().manual_seed(n)
    a = torch.randn(n, n + 3, dtype=torch.float64, generator=g)  # column-major, lda n + 3
    a[:, :n] += n * torch.eye(n, dtype=torch.float64)
    b = torch.randn(nrhs, n + 1, dtype=torch.float64, generator=g) * torch.logspace(-3, 3, nrhs)[:, None].double()
    da, x = a.cuda(), b.cuda()
    f = dp.Factor(n, da, n + 3, precision=dp.PRECISION_FP64)
    st, r = f.solve(x, n + 1, nrhs)
    assert st == dp.SUCCESS and r.backward_error <= 1e-14
    A, B, X = a[:, :n].numpy().T, b[:, :n].numpy().T, x.cpu().numpy()[:, :n].T
    den = np.abs(A).sum(axis=1).max() * np.abs(X).max(axis=0) + np.abs(B).max(axis=0)
    error = (np.abs(B - A @ X).max(axis=0) / den).max()
    assert abs(r.backward_error - error) <= 2 * (n + 2) * U  # either residual's own rounding
    assert torch.equal(x.cpu()[:, n:], b[:, n:])
