"""The kernels between two outer blocks at the edges of their tiles: the
trailing update on few tiles, bit for bit against the tile shape of large
updates (each element is one accumulator over k in order), and the block
inverse inside factorisations, by the backward error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0**-53


# 768 x 767 is below one 64 x 64 tile per SM, 900 x 769 above; one column to 33 beside
@pytest.mark.parametrize("m,n,k", [(1, 33, 5), (32, 32, 32), (33, 65, 31), (65, 33, 33), (200, 1, 100),
                                   (4097, 31, 64), (333, 37, 257), (768, 767, 64), (900, 769, 64)])
def test_update_on_few_tiles(built, m, n, k):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator().manual_seed(m * 7 + n)
    a, b, c = (torch.randn(*s, dtype=torch.float64, generator=g).cuda() for s in ((k, m), (n, k), (n, m)))
    out = []
    for tile in (0, 5):
        x = c.clone()
        previous = dp.gemm_tile(tile)
        try:
            dp.schur_update_device(m, n, k, a, m, b, k, x, m)
            torch.cuda.synchronize()
        finally:
            dp.gemm_tile(previous)
        out.append(x.cpu().numpy())
    assert out[0].tobytes() == out[1].tobytes()
    want = c.cpu().numpy() - b.cpu().numpy() @ a.cpu().numpy()
    bound = 2 * (k + 2) * U * (abs(b) @ abs(a) + abs(c)).cpu().numpy()
    assert (abs(out[0] - want) <= bound).all()


# outer blocks of w columns: solved by the inverse above 64, a warp and its remainders
@pytest.mark.parametrize("w", [65, 95, 96, 97, 128, 131, 223, 254, 256])
def test_block_inverse(built, w):
    import delayed_pivoting as dp
    import oracle as orc
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m, n = 2 * w + 70, 2 * w + 33
    a = np.asfortranarray(np.random.default_rng(w).standard_normal((m, n)))
    d = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    ip, jp = np.zeros(n, dtype=np.int32), np.zeros(n, dtype=np.int32)
    st, info = dp.getrf_device_ex(m, n, d, m, ip, jp, nb_outer=w)
    ri, rj, rinfo = orc.oracle_getrf(a.copy(order="F"))
    assert st == dp.SUCCESS and info == rinfo
    np.testing.assert_array_equal(ip, ri)
    np.testing.assert_array_equal(jp, rj)
    f = d.cpu().numpy().T
    p, q = np.arange(m), np.arange(n)
    for i in range(info):
        p[[i, ip[i]]] = p[[ip[i], i]]
        q[[i, jp[i]]] = q[[jp[i], i]]
    lower, upper = np.tril(f, -1)[:, :n] + np.eye(m, n), np.triu(f[:n])
    # U12 by inverse: |dU12| <= (w + 1) u (|T| |A12| + |A12|), |T| <= |L11^{-1}| |L11|-wise;
    # the updates add (n + 1) u |L| |U|
    t = max(np.abs(np.linalg.inv(lower[s:e, s:e])).sum(axis=1).max()
            for s, e in ((s, min(s + w, n)) for s in range(0, n, w)))
    bound = 2 * n * U * (1 + t) * (np.abs(lower) @ np.abs(upper)).max()
    assert np.abs(a[p][:, q] - lower @ upper).max() <= bound


def test_update_behind_others_and_under_capture(built):
    """A chain of updates, each reading what the one before wrote, is the same bits
    launched on a stream (each in place before the last has left) and replayed."""
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 96
    g = torch.Generator().manual_seed(1)
    a = (torch.randn(n, n, dtype=torch.float64, generator=g) / n).cuda()
    base = torch.randn(12, n, n, dtype=torch.float64, generator=g).cuda()

    def chain(x, stream):
        for i in range(1, 12):
            assert dp.schur_update_device(n, n, n, a, n, x[i - 1], n, x[i], n, stream=stream) == dp.SUCCESS

    direct, replayed = base.clone(), base.clone()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    chain(direct, s)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(replayed, torch.cuda.current_stream())
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(direct, replayed)
    want = base.cpu().numpy()
    for i in range(1, 12):
        want[i] -= want[i - 1] @ a.cpu().numpy()
    assert np.abs(direct.cpu().numpy() - want).max() <= 12 * (n + 2) * U * np.abs(want).max() * n
