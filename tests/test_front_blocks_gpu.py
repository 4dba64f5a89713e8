"""The solves of a front's two sides at the edges of their blocks (32 and 64
columns within 256), side by side and alone, on a stream of the caller's: records
and the whole front against the oracle, to the bound of the front tests."""
import numpy as np
import pytest

import oracle as orc
from test_front import make_front

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,p,tail,zc", [
    (256, 300, 256, 0, None), (300, 257, 257, 0, None), (290, 257, 256, 0, 9), (321, 322, 289, 1, None),
    (600, 640, 512, 0, 100), (700, 650, 545, 30, None), (900, 260, 257, 0, 0)])
def test_front_blocks(built, m, n, p, tail, zc):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    f = make_front(m, n, p, m + n, tail, zc)
    k0, ip0, jp0, out0 = orc.oracle_front(f, p)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        d = torch.from_numpy(np.ascontiguousarray(f.T)).cuda()
        rows, cols = np.arange(m, dtype=np.int32), np.arange(n, dtype=np.int32)
        st, k, ipiv, jpiv = dp.front_factor(m, n, p, d, m, rows, cols, stream=s)
    torch.cuda.synchronize()
    assert st == dp.SUCCESS and k == k0
    np.testing.assert_array_equal(ipiv, ip0)
    np.testing.assert_array_equal(jpiv, jp0)
    scale = max(1.0, float(np.abs(out0).max()))
    assert np.abs(d.cpu().numpy().T - out0).max() <= 1e-10 * scale * max(m, n) ** 0.5
