"""Large calls on a device that has little memory left.  A factorisation with room
for the FP64 updates' workspace (36 MB at n = 16384) but not for the integer
update's digits beside it (67 MB more) takes the FP64 updates; a solve with room for
its vectors but not for the buffers of 64 right-hand sides (25 MB at n = 24576)
takes them in narrower passes."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _device_left(dp, torch, mib):
    dp.lib().dp_memory_trim()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (mib << 20), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()
        dp.lib().dp_memory_trim()


def test_factorisation_without_room_for_the_digits(built):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 16384
    a = torch.randn(n, n, dtype=torch.float64, device="cuda",
                    generator=torch.Generator("cuda").manual_seed(2))
    w = torch.empty_like(a)

    def factor():
        ipiv, jpiv = np.zeros(n, dtype=np.int32), np.zeros(n, dtype=np.int32)
        w.copy_(a)
        torch.cuda.synchronize()
        return dp.getrf_device_ex(n, n, w, n, ipiv, jpiv), ipiv, jpiv

    want = factor()  # (and every kernel loaded)
    full = w.clone()
    with _device_left(dp, torch, 80):
        got = factor()
    assert want[0] == got[0] == (dp.SUCCESS, n)
    np.testing.assert_array_equal(want[1], got[1])
    np.testing.assert_array_equal(want[2], got[2])
    assert ((full - w).norm() / full.norm()).item() <= 1e-10


def test_solves_in_narrower_passes(built):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, nrhs = 24576, 64
    g = torch.Generator("cuda").manual_seed(3)
    a = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    b = torch.randn(nrhs, n, dtype=torch.float64, device="cuda", generator=g)
    f = dp.Factor(n, a, n, precision=dp.PRECISION_FP64)
    lu, ipiv, jpiv = a.clone(), np.zeros(n, dtype=np.int32), np.zeros(n, dtype=np.int32)
    assert dp.getrf_device_ex(n, n, lu, n, ipiv, jpiv) == (dp.SUCCESS, n)
    x, y = torch.empty_like(b), torch.empty_like(b)

    def solve():
        x.copy_(b)
        y.copy_(b)
        torch.cuda.synchronize()
        st, _ = f.solve(x, n, nrhs)
        return st, dp.getrs_device(n, nrhs, lu, n, ipiv, jpiv, y, n)

    assert solve() == (dp.SUCCESS, dp.SUCCESS)
    want = x.clone(), y.clone()
    with _device_left(dp, torch, 40):
        got = solve()
    f.close()
    assert got == (dp.SUCCESS, dp.SUCCESS)
    assert torch.equal(x, want[0]) and torch.equal(y, want[1])
