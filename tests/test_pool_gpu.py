"""The workspace and factor pools kept between calls: calls from several
threads on streams of their own give the results of one call alone, and the
memory kept is bounded and given back by dp_memory_trim."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lu(torch, dp, src, n, stream):
    with torch.cuda.stream(stream):
        d = src.clone()
    ipiv, jpiv = np.zeros(n, dtype=np.int32), np.zeros(n, dtype=np.int32)
    st, info = dp.getrf_device_ex(n, n, d, n, ipiv, jpiv, stream=stream)
    assert st == dp.SUCCESS and info == n
    return d.cpu(), ipiv, jpiv


def test_threads_and_streams_share_the_pools(built):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    orders = [90, 300, 700, 1100]
    src = [torch.randn(n, n, dtype=torch.float64, device="cuda",
                       generator=torch.Generator("cuda").manual_seed(n)) for n in orders]
    torch.cuda.synchronize()
    alone = [_lu(torch, dp, a, n, torch.cuda.Stream()) for a, n in zip(src, orders)]
    wrong = []

    def work(k):
        s = torch.cuda.Stream()
        for rep in range(6):
            i = (k + rep) % len(orders)
            got = _lu(torch, dp, src[i], orders[i], s)
            if not (torch.equal(got[0], alone[i][0]) and np.array_equal(got[1], alone[i][1])
                    and np.array_equal(got[2], alone[i][2])):
                wrong.append((k, rep))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong


def test_kept_memory_is_bounded_and_given_back(built):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 4096
    a = torch.randn(n, n, dtype=torch.float64, device="cuda")
    dp.Factor(n, a, n).close()  # library and context set up
    dp.lib().dp_memory_trim()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    live = [dp.Factor(n, a, n, precision=dp.PRECISION_FP64) for _ in range(40)]  # 5.4 GB
    for f in live:
        f.close()
    torch.cuda.synchronize()
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert kept <= (4 << 30) + (256 << 20)
    dp.lib().dp_memory_trim()
    assert free0 - torch.cuda.mem_get_info()[0] <= 256 << 20
