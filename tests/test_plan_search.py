"""The plan search at sizes where its sampled sums run over several batches of the kernel that
replays the reference's serial float sum: against the oracle, on smooth data, data with exact
zeros and rounding ties (few significant bits), and counts around a batch's 8192 terms."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["smooth", "ties", "zeros", "rough"])
@pytest.mark.parametrize("shape", [(64, 80, 80), (96, 100, 121)], ids=["one-batch", "several"])
def test_sampled_sums_against_oracle(gpu_ctx, kind, shape):
    import asz_b200.api as api
    from asz_b200 import fields
    rng = np.random.default_rng(5)
    f = fields.grf_field(shape, 1.5 if kind == "rough" else 3.5, rng).astype(np.float32)
    eb = 1e-3
    if kind == "ties":
        f, eb = np.round(f * 64) / 64, 2.0 ** -9
    elif kind == "zeros":
        f[: shape[0] // 2] = 0.0
    f = f.astype(np.float32)
    o = O.compress(f, eb, None, False, O.default_params(block_pivot_ratio=3))
    blob, rep = gpu_ctx.compress(f, eb, None, "cubic", api.default_params(block_pivot_ratio=3))
    assert [rep.plan_best_dist[k] for k in range(rep.plan_search_layers)] == list(o.best_dist)
    assert rep.plan.decode() == o.plan
    assert blob == o.asz
