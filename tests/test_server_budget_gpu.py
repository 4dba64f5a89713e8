"""The server's budget at its edge: a factorisation that is accepted with room for
its own solve serves its follow-ups in that room too, one by one, and more is never
in use than the budget."""
import time

import pytest

pytestmark = pytest.mark.gpu


def _torch():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _least_budget(dp, n, nrhs, d_a, d_b):
    """The smallest budget a request of this size is accepted with."""
    lo, hi = 1, 1 << 28  # refused, accepted
    while hi - lo > 1:
        mid = (lo + hi) // 2
        s = dp.Server(budget_bytes=mid, large_workers=1)
        if s.submit(1, n, d_a, n, d_b, n, nrhs) == 0:
            hi = mid
        else:
            lo = mid
        s.close()
    return hi


@pytest.mark.parametrize("n,nrhs,spare", [(100, 8, 0), (600, 8, 0), (600, 8, 2000), (600, 32, 600 * 32 * 8),
                                          (600, 8, 600 * 8 * 36)])
def test_follow_ups_run_beside_the_factor(built, n, nrhs, spare):
    import delayed_pivoting as dp

    torch = _torch()
    g = torch.Generator(device="cuda").manual_seed(n + nrhs)
    a = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    a += 2 * n ** 0.5 * torch.eye(n, dtype=torch.float64, device="cuda")
    x = [torch.randn(nrhs, n, dtype=torch.float64, device="cuda", generator=g) for _ in range(3)]
    b = [v @ a for v in x]
    torch.cuda.synchronize()
    budget = _least_budget(dp, n, nrhs, a, torch.zeros_like(b[0])) + spare
    s = dp.Server(budget_bytes=budget, large_workers=2)
    assert s.submit(1, n, a, n, b[0], n, nrhs, followups=2) == 0
    for i in (1, 2):
        assert s.submit(1 + i, n, None, n, b[i], n, nrhs, factor_id=1) == 0
    done = {}
    t0 = time.time()
    while len(done) < 3 and time.time() - t0 < 20:
        for r in s.poll(8, wait_ms=50):
            done[r.id] = r
    stats = s.stats()
    s.close()
    assert sorted(done) == [1, 2, 3]
    assert all(r.status == 0 and r.backward_error <= 1e-14 for r in done.values())
    for v, got in zip(x, b):
        assert (got - v).abs().max().item() <= 1e-9 * v.abs().max().item()
    assert stats.bytes_peak <= budget and stats.residents == 0
