"""The sweep's 32-bit QBs and their 64-bit repeat, several coefficients a thread, and streams that are
encoded and copied out alone or together, against the CPU oracle."""
import numpy as np
import pytest

import oracle as O

SUM_RTOL = 1e-12


def _streams_equal(rows, d, pred, mode):
    """The figures that the QB streams alone give; returns the oracle's rows."""
    exp = [O.sweep_run(d, pred, r.rel_eb, r.c0, r.c1, mode) for r in rows]
    for r, o in zip(rows, exp):
        assert (r.samples, r.huffman_bytes, r.zstd_bytes) == (o.samples, o.huffman_bytes, o.zstd_bytes)
        assert (r.br, r.cr, r.h1) == (o.br, o.cr, o.h1)
    return exp


@pytest.mark.gpu
@pytest.mark.parametrize("pred,mode", [("1d4r0_xx0", "legacy"), ("2d4r01_xx2", "common"), ("1d6r0_xx1", "legacy")])
def test_wide_bins(gpu_ctx, pred, mode):
    """A field curved along axis 0 at a bound of 1e-12: bins beyond 2^31 for the coefficients that
    miss the curvature, in a narrow range. The next bound, 1e-3, fits 32 bits again."""
    from asz_b200 import sweep
    rng = np.random.default_rng(3)
    d = (np.arange(14.0) ** 2)[:, None, None] + 1e-4 * rng.integers(0, 9, (14, 17, 13))
    d = d.astype(np.float32)
    rows, _ = sweep.run(gpu_ctx, d, pred, [1e-12, 1e-3], mode, "legacy")
    assert len(rows) == 2 * len(sweep.coefficients(pred, "legacy"))
    for r, o in zip(rows, _streams_equal(rows, d, pred, mode)):
        for a, b in ((r.mse_sum, o.mse_sum), (r.rmse_sum, o.rmse_sum), (r.mae_sum, o.mae_sum)):
            assert abs(a - b) <= SUM_RTOL * abs(b)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,pred", [((90, 300, 330), "1d4r2_xx2"), ((130, 200, 340), "2d4r02_xx0")])
def test_streams_alone(gpu_ctx, shape, pred):
    """Streams of more than 2^22 symbols go through encoding and copying one by one (their sums, which
    do not, have millions of terms, and the oracle's serial ones are too far off to compare with)."""
    from asz_b200 import fields, sweep
    d = np.ascontiguousarray(fields.grf_field(shape, 3.0, np.random.default_rng(5)), dtype=np.float32)
    rows, _ = sweep.run(gpu_ctx, d, pred, [1e-3], "legacy", "legacy")
    _streams_equal([rows[0], rows[-1]], d, pred, "legacy")
