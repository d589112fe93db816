"""Two threads with a context each, on fields whose coefficient groups, codes and lines ask the same
kernels for different amounts of shared memory: each gets the streams and values it gets alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_threads():
    import asz_b200.api as api
    from asz_b200 import fields
    rng = np.random.default_rng(5)
    mixed = ",".join(["cubic0_012", "cubic1_120", "cubic2_021"] * 2)
    jobs = [((40, 44, 48), 1e-3, mixed, 256), ((36, 40, 64), 1e-5, ",".join(["cubic2_012"] * 5), 64)]
    fs = [fields.grf_field(s, 2.5, rng).astype(np.float32) for s, *_ in jobs]

    def once(ctx, k):
        shape, eb, plan, samples = jobs[k]
        p = api.default_params(block_pivot_ratio=3, h1_block_sampling_num=samples)
        blob, _ = ctx.compress(fs[k], eb, plan, "cubic", p)
        both = ctx.compress_batch([fs[k], fs[k][1:]], eb, plan, "cubic", p)[0]
        return blob, [bytes(b) for b in both], ctx.decompress(blob, shape, eb, p)[0]

    want, bad = [], []
    for k in range(2):
        ctx = api.Context()
        ctx.set_tsel_mode(1)
        want.append(once(ctx, k))

    def work(k):
        try:
            ctx = api.Context()
            ctx.set_tsel_mode(1)
            for _ in range(25):
                blob, both, out = once(ctx, k)
                if blob != want[k][0] or both != want[k][1] or not np.array_equal(out, want[k][2]):
                    bad.append((k, "differs"))
        except Exception as e:  # noqa: BLE001 - reported below
            bad.append((k, repr(e)))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(300)
    assert not bad
