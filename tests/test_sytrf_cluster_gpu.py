"""The Bunch-Kaufman panel in one cluster against the same panel on a cooperative
grid: factors, records and near-tie counts bit for bit, at the edges of a CTA's
rows, of the cluster sizes and of the rows a cluster holds (4096: beyond, the
first panels use the grid), with delays, ties, zeros and non-finite entries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kind", [(1, "plain"), (2, "plain"), (127, "delays"), (129, "plain"),
                                    (257, "ties"), (300, "nan"), (520, "zero"), (1025, "delays"),
                                    (2049, "plain"), (2200, "ties"), (4160, "plain")])
def test_cluster_equals_grid(n, kind):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    if kind == "ties":
        a = np.sign(a)
    elif kind == "zero":
        a[:] = 0.0
    elif kind == "delays":
        idx = rng.choice(n, 9, replace=False)
        a[idx] = a[:, idx] = 0.0
        a[np.ix_(idx[:4], idx[4:8])] = 1e-17
    elif kind == "nan":
        a[n // 2, n // 3] = np.nan
        a[n - 1, 5] = np.inf
    a = torch.from_numpy(np.tril(a) + np.tril(a, -1).T).cuda()
    out = []
    for grid in (0, (n + 127) // 128):
        f = a.clone()
        st, perm, piv, info = dp.sytrf_device(n, f, n, grid=grid)
        r = dp.sytrf_last_report()
        lower = torch.triu(f).cpu().numpy().view(np.int64)  # (column-major: the lower triangle)
        out.append((st, info, perm.tobytes(), piv.tobytes(), lower.tobytes(),
                    tuple(r[x] for x in ("decisions", "near_ties", "max_closeness"))))
    assert out[0] == out[1]
    assert out[0][0] == dp.SUCCESS
