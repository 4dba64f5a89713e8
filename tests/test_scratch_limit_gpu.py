"""A large factorisation on a device with room for the FP64 updates' workspace (36 MB
at n = 16384) but not for the integer update's digits beside it (67 MB more): it
takes the FP64 updates instead of failing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
    dp.lib().dp_memory_trim()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (80 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = factor()
    finally:
        del hog
        torch.cuda.empty_cache()
        dp.lib().dp_memory_trim()
    assert want[0] == got[0] == (dp.SUCCESS, n)
    np.testing.assert_array_equal(want[1], got[1])
    np.testing.assert_array_equal(want[2], got[2])
    assert ((full - w).norm() / full.norm()).item() <= 1e-10
