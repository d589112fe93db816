"""The exact coefficient replay at the sizes where it changes form: groups of few samples (one warp's
rehash stages), around the bucket counts of the map's growth, more nodes than the CTA has threads,
more than the side-by-side tables or shared memory hold, on data with many equal keys, ties of the
float sums and wide errors; every group goes through the replay (selection mode 1)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _field(kind, shape, rng):
    from asz_b200 import fields
    if kind == "noise":
        f = rng.random(shape)
    elif kind == "steps":  # few significant bits: equal keys, sums that tie
        f = np.round(fields.grf_field(shape, 3.0, rng) * 32) / 32
    else:
        f = fields.grf_field(shape, 2.0, rng)
        f[: shape[0] // 3] = 0.0
    return f.astype(np.float32)


@pytest.mark.parametrize("kind", ["noise", "steps", "zeros"])
@pytest.mark.parametrize("samples", [20, 60, 256, 700, 1500, 3000, 6000])
def test_group_sizes_against_oracle(gpu_ctx, kind, samples):
    import asz_b200.api as api
    rng = np.random.default_rng(samples)
    f = _field(kind, (34, 37, 52), rng)
    plan = ",".join(["cubic0_012", "cubic1_120", "cubic2_021"] * 2)
    p = dict(block_pivot_ratio=4, h1_block_sampling_num=samples)
    o = O.compress(f, 1e-3, plan, False, O.default_params(**p))
    gpu_ctx.set_tsel_mode(1)
    try:
        blob, rep = gpu_ctx.compress(f, 1e-3, plan, "cubic", api.default_params(**p))
    finally:
        gpu_ctx.set_tsel_mode(0)
    assert np.float32(rep.default_slope) == np.float32(o.default_slope)
    assert np.array_equal(gpu_ctx.debug_t(), o.t_int)
    assert blob == o.asz
