"""The server's kernels for small requests at the edges of their blocks: orders
around the 32-row diagonal blocks, the 64-row residual tiles and the 256 threads,
right-hand sides around the eight of a solving CTA and the 32 of a residual pass,
padded leading dimensions, all in one burst."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0**-53


@pytest.mark.parametrize("tol", [1e-14, 1e-17])  # the second refines until it stalls
def test_small_requests(tol):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(5)
    shapes = [(n, k) for n in (1, 2, 31, 32, 33, 63, 64, 65, 255, 288, 289, 511, 512)
              for k in ((1, 9) if n < 200 else (7, 8, 33, 64))]
    srv = dp.Server(tol=tol)
    calls = []
    for rid, (n, k) in enumerate(shapes, 1):
        lda, ldb = n + rid % 3, n + rid % 2
        a = rng.standard_normal((n, n)) + 3.0 * np.eye(n)
        b = rng.standard_normal((n, k)) * 10.0 ** rng.uniform(-3, 3, (1, k))
        da, db = np.full((n, lda), 7.0), np.full((k, ldb), 7.0)
        da[:, :n], db[:, :n] = a.T, b.T
        calls.append((rid, n, k, a, b, torch.from_numpy(da).cuda(), lda, torch.from_numpy(db).cuda(), ldb))
    torch.cuda.synchronize()
    for rid, n, k, a, b, da, lda, db, ldb in calls:
        assert srv.submit(rid, n, da, lda, db, ldb, k) == 0
    results = {}
    while len(results) < len(calls):
        for r in srv.poll(256, wait_ms=1000):
            results[r.id] = r
    srv.close()
    for rid, n, k, a, b, da, lda, db, ldb in calls:
        r, x = results[rid], db.cpu().numpy()[:, :n].T
        assert r.status == 0 and r.info == n
        res = np.abs(b - (a.astype(np.longdouble) @ x.astype(np.longdouble))).max(axis=0)
        den = np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0)
        error = float((res / den).max())
        # the reported error: the residual in working precision, (n + 2) u relative to den
        assert abs(r.backward_error - error) <= (n + 2) * U * (1 + 1e-10)
        assert r.backward_error <= 1e-14 and (tol == 1e-14 or n == 1 or r.iterations > 0)
        if ldb > n:
            assert (db.cpu().numpy()[:, n:] == 7.0).all()
