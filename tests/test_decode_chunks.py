"""Decoding in short chunks (256 bits, 24 to a warp, 192 to a CTA): streams of less than a chunk up to
several CTAs' tiles, steep codes and spread ones, and streams that keep the long chunks (nearly
even code lengths, many bits a symbol). The decoded field is the oracle's to the bit."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eb", [3e-2, 1e-3, 3e-5])
@pytest.mark.parametrize("shape", [(7, 8, 9), (12, 13, 14), (21, 22, 23), (37, 38, 39), (60, 61, 62), (97, 98, 99)])
def test_against_oracle(gpu_ctx, shape, eb):
    import asz_b200.api as api
    from asz_b200 import fields
    rng = np.random.default_rng(sum(shape))
    f = fields.grf_field(shape, 2.5, rng)
    f[rng.random(shape) < 0.01] *= 3  # a few rare symbols: long codes
    f = f.astype(np.float32)
    plan = ",".join(["cubic0_012", "cubic1_120", "cubic2_021"] * 2)
    p = O.default_params(block_pivot_ratio=3)
    o = O.compress(f, eb, plan, False, p)
    want = O.decompress(o.asz, shape, eb, p)
    got, _ = gpu_ctx.decompress(o.asz, shape, eb, api.default_params(block_pivot_ratio=3))
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
