"""A batch's ranges, default slopes and histograms, each taken in one launch for all fields: fields that
go their own way there among others that do not (a zero extremum, few samples, a step too fine for
the replay's keys), starts at every alignment, streams of few and of many symbols. Each
field's stream is the one that compressing it alone gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fields(rng):
    from asz_b200 import fields
    f = [fields.grf_field(s, 2.5, rng).astype(np.float32) for s in [(9, 10, 11), (21, 30, 25), (40, 33, 57), (64, 17, 31)]]
    f.append(np.maximum(fields.grf_field((20, 31, 22), 3.0, rng), 0).astype(np.float32))  # zero minimum
    f.append(np.minimum(fields.grf_field((23, 20, 24), 3.0, rng), -0.0).astype(np.float32))  # zero maximum
    f.append((1e4 * fields.grf_field((33, 34, 35), 2.0, rng)).astype(np.float32))
    return f


@pytest.mark.parametrize("eb,kw", [(1e-2, {}), (1e-5, {}), (1e-3, dict(stat_eb_ratio=1e-8)), (1e-3, dict(h1_block_sampling_num=6000))])
@pytest.mark.parametrize("start", [None, 0, 1, 2, 3])  # None: host fields
def test_as_alone(gpu_ctx, eb, kw, start):
    import torch
    import asz_b200.api as api
    p = api.default_params(block_pivot_ratio=3, **kw)
    plan = ",".join(["cubic0_012", "cubic1_120", "cubic2_021"] * 2)
    fs = _fields(np.random.default_rng(7))
    want = [gpu_ctx.compress(f, eb, plan, "cubic", p)[0] for f in fs]
    given = fs
    if start is not None:  # packed one after another, so that the later starts vary too
        flat = torch.zeros(start + sum(f.size for f in fs), device="cuda")
        given, at = [], start
        for f in fs:
            given.append(flat[at : at + f.size].view(f.shape))
            given[-1].copy_(torch.from_numpy(f))
            at += f.size
        torch.cuda.synchronize()
    got = gpu_ctx.compress_batch(given, eb, plan, "cubic", p)[0]
    assert [bytes(g) for g in got] == [bytes(w) for w in want]


@pytest.mark.parametrize("bad,match", [("nan", "field 2: input contains a nonfinite value"), ("same", "field 2: max_val==min_val")])
def test_errors_name_the_field(gpu_ctx, bad, match):
    import asz_b200.api as api
    fs = _fields(np.random.default_rng(8))
    fs[2] = np.full_like(fs[2], 3.0) if bad == "same" else fs[2].copy()
    if bad == "nan":
        fs[2].flat[17] = np.nan
    with pytest.raises(api.AszError, match=match):
        gpu_ctx.compress_batch(fs, 1e-3, "cubic0_012,cubic1_120,cubic2_021", "cubic", api.default_params(block_pivot_ratio=3))
