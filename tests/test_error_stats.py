"""asz_error_stats_noalloc at the edges of its tiles and vector loads: lengths around 4096 and 8192
values, arrays off a 16-byte boundary (one or both), against float64 on the host."""
import numpy as np
import pytest

import asz_b200.api as api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4095, 4096, 4097, 8191, 8192, 8193, 3 * 65536 + 5])
@pytest.mark.parametrize("off", [(0, 0), (1, 0), (3, 3)])
def test_lengths_and_alignment(n, off):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n + 4, generator=g, device="cuda")[off[0]: off[0] + n]
    y = torch.randn(n + 4, generator=g, device="cuda")[off[1]: off[1] + n]
    y[n - 1] = x[n - 1] + 20.0  # the last value decides the maximum
    torch.cuda.synchronize()
    m, p = api.error_stats_noalloc(x, y, 3.0)
    xh, yh = x.cpu().numpy(), y.cpu().numpy()
    d = xh.astype(np.float64) - yh.astype(np.float64)
    assert m == float(np.abs(xh - yh).max())
    # n additions of non-negative doubles in any order: relative error below n 2^-53 each way.
    ref = 10 * np.log10(9.0 / np.mean(d * d))
    assert abs(p - ref) <= 10 / np.log(10) * (2 * n + 8) * 2.0 ** -53 + 4e-15 * abs(ref)


@pytest.mark.parametrize("n", [4096, 70000, 1 << 21])
def test_same_bits_at_any_alignment(n):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    for _ in range(8):
        x, y = torch.randn(n, generator=g, device="cuda"), torch.randn(n, generator=g, device="cuda")
        got = []
        for off in [(0, 0), (1, 1), (0, 3), (2, 0)]:
            a, b = (torch.empty(n + 4, device="cuda")[o: o + n].copy_(v) for o, v in zip(off, (x, y)))
            torch.cuda.synchronize()
            got.append(api.error_stats_noalloc(a, b, 3.0))
        assert len(set(got)) == 1, got
