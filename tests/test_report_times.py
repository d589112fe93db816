"""What a call's times and profile entries hold: decoding and reconstruction apart in a decompression's
report, and an entry for every kernel of the plan search and of the predictor-family selection."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Entry(C.Structure):
    _fields_ = [("name", C.c_char * 32), ("launches", C.c_uint64), ("ms", C.c_double), ("bytes", C.c_uint64)]


def _profiled(ctx, call):
    entries = (Entry * 64)()
    ctx._L.asz_profile_enable(ctx._c, 1)
    ctx._L.asz_profile_read(ctx._c, entries, 64, 1)
    try:
        call()
        n = ctx._L.asz_profile_read(ctx._c, entries, 64, 1)
    finally:
        ctx._L.asz_profile_enable(ctx._c, 0)
    return {e.name.decode(): e for e in entries[:n]}


def test_decompression_times(gpu_ctx):
    import torch
    import asz_b200.api as api
    from asz_b200 import fields
    f = fields.grf_field((256, 320, 320), 11 / 3, np.random.default_rng(3)).astype(np.float32)
    p = api.default_params(block_pivot_ratio=3)
    blob, _ = gpu_ctx.compress(f, 1e-4, ",".join(["cubic2_012"] * 7), "cubic", p)
    out = torch.empty(f.shape, device="cuda")
    reps = [gpu_ctx.decompress(blob, f.shape, 1e-4, p, out=out)[1] for _ in range(9)][1:]
    prof = _profiled(gpu_ctx, lambda: gpu_ctx.decompress(blob, f.shape, 1e-4, p, out=out))
    writing = prof["huff_decode_write"].ms / 1e3
    rebuilding = sum(e.ms for k, e in prof.items() if k.endswith("_decompress")) / 1e3
    assert min(r.core_s for r in reps) < rebuilding + writing / 2
    for r in reps:
        assert r.huffman_s > writing + prof["huff_decode_sync"].ms / 1e3
        assert r.zstd_s + r.h2d_s + r.core_s < r.total_s and r.huffman_s + r.core_s < r.total_s


def test_profile_has_every_kernel(gpu_ctx):
    """The plan search and the family probes (their bytes: what a kernel reads and writes at least)."""
    import asz_b200.api as api
    from asz_b200 import fields
    f = fields.grf_field((60, 150, 170), 3.0, np.random.default_rng(4)).astype(np.float32)
    p = api.default_params(block_pivot_ratio=3)
    plan = "cubic0_012,cubic1_120,cubic2_021"
    run = {fam: _profiled(gpu_ctx, lambda: gpu_ctx.compress(f, 1e-3, plan, fam, p)) for fam in ("cubic", "auto")}
    # The probes' kernels are the rounds' own, with their bytes, and the gather of their targets.
    for k in ("pivot_compress", "tsel_fast", "round_compress"):
        assert run["auto"][k].launches > run["cubic"][k].launches, k
        assert run["auto"][k].bytes > run["cubic"][k].bytes, k
    assert run["auto"]["probe_points"].launches > 0 and run["auto"]["probe_points"].ms > 0
    got = _profiled(gpu_ctx, lambda: gpu_ctx.compress(f, 1e-3, None, "cubic", p))
    layers = got["plan_sample"].launches
    assert layers > 3 and got["plan_mse"].launches == layers and got["plan_mse"].ms > 0
    # A QB and an error written of each sample, and the error read again.
    assert got["plan_sample"].bytes == 2 * got["plan_mse"].bytes
