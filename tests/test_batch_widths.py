"""Panel widths of the batched factorisation: the defaults and the autotuner name
widths that the kernels run (their windows hold 16 columns), and wider ones are
taken as 16, with the same bits."""
import numpy as np
import pytest

WINDOW = 16


def test_defaults_are_widths_that_run(built):
    import delayed_pivoting as dp

    assert all(1 <= v <= WINDOW for v in dp.batch_options().nb_bucket)


@pytest.mark.gpu
def test_autotuner_times_widths_that_run(built):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    for seed in range(4):
        st, opt = dp.batch_autotune(samples=6, seed=seed)
        assert st == dp.SUCCESS and all(1 <= v <= WINDOW for v in opt.nb_bucket)


@pytest.mark.gpu
def test_wider_than_the_window_is_the_window(built):
    import delayed_pivoting as dp
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ns = [40, 100, 200, 400]
    out = []
    for nb in (WINDOW, 24, 32):
        b = dp.Batch(ns, options=dp.batch_options(nb_bucket=nb))
        base = torch.randn(b.total_elements, dtype=torch.float64, device="cuda",
                           generator=torch.Generator("cuda").manual_seed(4))
        ip, jp = (torch.zeros(b.total_records, dtype=torch.int32, device="cuda") for _ in range(2))
        info = torch.zeros(len(ns), dtype=torch.int32, device="cuda")
        assert b.getrf_async(base, ip, jp, info) == dp.SUCCESS
        torch.cuda.synchronize()
        out.append([t.cpu().numpy() for t in (base, ip, jp, info)])
        b.close()
    for other in out[1:]:
        for x, y in zip(out[0], other):
            np.testing.assert_array_equal(x, y)
