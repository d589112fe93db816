"""Decompression of consecutive rounds along axis 2 in one launch: runs at the plan's start, middle and
end, every QB order, lines shorter and longer than a chunk of targets, one and many blocks along the
axis, lines that leave a CTA few warps and lines too long for the launch, rounds without targets."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

CASES = [
    ((9, 10, 16), "cubic2_012", 4, 1),
    ((9, 10, 17), "cubic2_120", 4, 3),
    ((9, 8, 33), "cubic2_021", 7, 3),
    ((20, 23, 129), "cubic2_012", 9, 3),
    ((20, 23, 131), "cubic2_120,cubic2_012,cubic2_021", 2, 1),
    ((24, 20, 95), "cubic0_012,cubic2_120,cubic2_021,cubic1_120,cubic2_012,cubic2_012,cubic2_012", 1, 2),
    ((12, 11, 300), "cubic2_012,cubic2_021,cubic0_012,cubic1_120", 1, 1),
    ((9, 8, 1000), "cubic2_012", 3, 1),
    ((9, 8, 7001), "cubic2_012", 12, 3),
    ((9, 8, 17000), "cubic2_012", 4, 3),
    ((9, 8, 30000), "cubic2_012", 5, 3),
]


@pytest.mark.parametrize("family", ["cubic", "quintic"])
@pytest.mark.parametrize("shape,rounds,times,bpr", CASES)
def test_against_oracle(gpu_ctx, shape, rounds, times, bpr, family):
    import asz_b200.api as api
    from asz_b200 import fields
    plan = ",".join([rounds] * times)
    f = fields.grf_field(shape, 2.0, np.random.default_rng(sum(shape))).astype(np.float32)
    p = O.default_params(block_pivot_ratio=bpr)
    o = O.compress(f, 1e-3, plan, family == "quintic", p)
    want = O.decompress(o.asz, shape, 1e-3, p)
    got, _ = gpu_ctx.decompress(o.asz, shape, 1e-3, api.default_params(block_pivot_ratio=bpr))
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
