"""Huffman decoding where its synchronisation is put to the test: streams of codes of one length, which
never resynchronise from a wrong guess (5 and 7 bits against chunks of 1024), of two lengths, and of a
steep code; lengths around a chunk, a tile of chunks and several tiles. The values are uniform noise
on a lattice, so the finest round's symbols are spread as chosen."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [2, 3, 32, 128, 100])
@pytest.mark.parametrize("shape", [(7, 8, 9), (16, 20, 24), (40, 48, 60), (64, 96, 128)])
def test_even_codes_round_trip(gpu_ctx, levels, shape):
    import asz_b200.api as api
    rng = np.random.default_rng(levels)
    f = rng.integers(0, levels, size=shape).astype(np.float32)
    f.flat[0], f.flat[1] = 0, max(levels - 1, 1)
    p = api.default_params(block_pivot_ratio=3, eb_ratio=1.0)
    eb = 0.49 / max(levels - 1, 1)
    blob, rep = gpu_ctx.compress(f, eb, "cubic2_012", "cubic", p)
    o = O.compress(f, eb, "cubic2_012", False, O.default_params(block_pivot_ratio=3, eb_ratio=1.0))
    assert blob == o.asz
    for _ in range(2):  # the second call finds the first one's arrays
        dec, _ = gpu_ctx.decompress(blob, f.shape, eb, p)
        assert np.array_equal(dec.view(np.uint32), o.recon.view(np.uint32))
