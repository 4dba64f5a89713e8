"""The batched factorisation at the edges of its size classes, and with so many
exact-zero columns that the row moves owed to the finished columns outgrow the
lists they are kept in: records and residuals against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 15, 16, 17, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 400, 511, 512]


def _run(dp, torch, mats, graph):
    plan = dp.Batch([a.shape[0] for a in mats])
    host = np.zeros(plan.total_elements)
    for a, o in zip(mats, plan.offsets):
        host[o:o + a.size] = a.T.reshape(-1)
    base = torch.from_numpy(host).cuda()
    ipiv = torch.empty(plan.total_records, dtype=torch.int32, device="cuda")
    jpiv, info = torch.empty_like(ipiv), torch.empty(len(mats), dtype=torch.int32, device="cuda")
    call = plan.getrf_graph if graph else plan.getrf_async
    assert call(base, ipiv, jpiv, info) == dp.SUCCESS
    report = plan.last_report()
    out, ipiv, jpiv, info = (t.cpu().numpy() for t in (base, ipiv, jpiv, info))
    for a, o, r, k in zip(mats, plan.offsets, plan.record_offsets, info):
        n = a.shape[0]
        yield a, out[o:o + n * n].reshape(n, n).T, ipiv[r:r + n], jpiv[r:r + n], int(k), report


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("zeros", [0, 1, 40])
def test_class_edges(built, zeros, graph):
    import delayed_pivoting as dp
    import oracle as orc
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    mats = []
    for i, n in enumerate(ORDERS):
        rng = np.random.default_rng(31 * n + zeros)
        a = rng.standard_normal((n, n))
        a[:, rng.choice(n, min(n, zeros * n // 128 + (zeros > 0)), replace=False)] = 0.0
        mats.append(a)
    for a, f, ip, jp, k, report in _run(dp, torch, mats, graph):
        n = a.shape[0]
        ref = np.asfortranarray(a)
        ri, rj, rinfo = orc.oracle_getrf(ref)
        assert report["near_ties"] == 0 and k == rinfo
        np.testing.assert_array_equal(ip, ri)
        np.testing.assert_array_equal(jp, rj)
        if k:
            assert orc.scaled_residual(np.asfortranarray(a), np.asfortranarray(f), n, n, k, ip, jp) <= 10.0
        else:
            assert not f.any()
