"""The predictor-family probes as one batch of frames and frame by frame, where both are taken: one
target and many, more targets than a batch holds, blocks cut by the field's far faces, and rounds whose
targets' spans are empty or of one point. Both forms give the oracle's figures to the last bit."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

FIGURES = ("fam_cubic_mse", "fam_quintic_mse", "fam_cubic_psnr", "fam_quintic_psnr", "fam_cubic_h1", "fam_quintic_h1",
           "fam_score_gain")


@pytest.mark.parametrize("shape,eb,targets,suffix", [
    ((41, 37, 53), 1e-3, 1, 6),
    ((41, 37, 53), 1e-4, 24, 6),
    ((33, 40, 47), 1e-2, 400, 3),
    ((9, 70, 31), 1e-3, 8, 1),
    ((64, 64, 64), 1e-5, 8, 9),
])
def test_forms_against_oracle(gpu_ctx, shape, eb, targets, suffix):
    import asz_b200.api as api
    from asz_b200 import fields
    f = fields.grf_field(shape, 2.5, np.random.default_rng(sum(shape))).astype(np.float32)
    plan = ",".join(["cubic0_012", "cubic1_120", "cubic2_021"] * 3)
    kw = dict(block_pivot_ratio=3, predictor_family_sample_blocks=targets, predictor_family_sample_fraction_limit=1.0,
              predictor_family_suffix_layers=suffix)
    o = O.compress(f, eb, plan, None, O.default_params(**kw))
    for mode in (0, 1):  # 1: every group through the exact replay, frame by frame
        gpu_ctx.set_tsel_mode(mode)
        try:
            blob, rep = gpu_ctx.compress(f, eb, plan, "auto", api.default_params(**kw))
        finally:
            gpu_ctx.set_tsel_mode(0)
        for k in ("fam_blocks", "fam_points") + FIGURES:
            assert getattr(rep, k) == o.family[k], (mode, k)
        assert bool(rep.quintic) == o.quintic and blob == o.asz
