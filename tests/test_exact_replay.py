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


@pytest.mark.parametrize("family", ["cubic", "quintic"])
def test_keys_beyond_int32(gpu_ctx, family):
    """A statistics step so fine that the samples' keys leave int32: of those groups, the ones that reach
    the exact replay (all of them in selection mode 1) go to the serial kernel, for which the rounds
    are repeated."""
    import asz_b200.api as api
    from asz_b200 import fields
    rng = np.random.default_rng(17)
    fs = [fields.grf_field(s, 2.5, rng).astype(np.float32) for s in [(20, 22, 26), (18, 25, 31)]]
    plan = ",".join(["cubic0_012", "cubic1_120", "cubic2_021"] * 2)
    kw = dict(block_pivot_ratio=3, stat_eb_ratio=1e-8)
    p = api.default_params(**kw)
    want = [O.compress(f, 1e-3, plan, family == "quintic", O.default_params(**kw)) for f in fs]
    for mode in (1, 0):
        for f, o in zip(fs, want):
            gpu_ctx.set_tsel_mode(mode)
            try:
                blob, rep = gpu_ctx.compress(f, 1e-3, plan, family, p)
            finally:
                gpu_ctx.set_tsel_mode(0)
            assert rep.serial_groups > 0 or mode == 0
            assert np.array_equal(gpu_ctx.debug_t(), o.t_int)
            assert blob == o.asz
    for _ in range(2):
        blobs, _, _ = gpu_ctx.compress_batch(fs, 1e-3, plan, family, p)
        assert blobs == [o.asz for o in want]
