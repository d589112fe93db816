"""Payloads encoded at their places in the assembled stream: any byte offset within a word, streams
that end within a word of the next header, single-symbol streams without a payload."""
import numpy as np
import pytest

import oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("shape,layers", [((16, 16, 16), 3), ((17, 19, 23), 3), ((33, 40, 52), 5)])
@pytest.mark.parametrize("eb", [0.3, 1e-2, 1e-5])
def test_places(gpu_ctx, shape, layers, eb):
    import asz_b200.api as api
    rng = np.random.default_rng(int(1 / eb) + layers)
    f = np.cumsum(rng.standard_normal(shape), axis=2).astype(np.float32)
    for k in range(2, layers + 1):  # headers of 9 + 2 k bytes: the payloads' offsets move by two
        plan = ",".join(["cubic2_012"] * k)
        p = api.default_params(block_pivot_ratio=3)
        blob, _ = gpu_ctx.compress(f, eb, plan, "cubic", p)
        assert blob == O.compress(f, eb, plan, False, O.default_params(block_pivot_ratio=3)).asz


@pytest.mark.gpu
def test_fields_side_by_side(gpu_ctx):
    """Fields of a batch lie in one image: each equals its single call."""
    import asz_b200.api as api
    rng = np.random.default_rng(11)
    plan = "cubic2_012,cubic1_120,cubic0_012"
    p = api.default_params(block_pivot_ratio=3)
    fields = [np.cumsum(rng.standard_normal((16 + i, 18 + 3 * i, 17 + 5 * i)), axis=1).astype(np.float32) for i in range(11)]
    blobs, _, _ = gpu_ctx.compress_batch(fields, 1e-3, plan, "cubic", p)
    assert [bytes(b) for b in blobs] == [gpu_ctx.compress(f, 1e-3, plan, "cubic", p)[0] for f in fields]
