"""The relaxed proxy's forward and backward kernels over the group sizes where they change form: empty,
below and above a warp and its unrolled pass, up to and beyond the largest group a warp takes.
Samples keep a tenth of a bin away from its edges, so rounding moves no sample to another bin."""
import numpy as np
import pytest
import torch

from asz_b200.grad import EPS, relaxed_proxy_torch

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 2, 3, 31, 32, 33, 127, 128, 129, 1023, 1024, 1560, 4095, 4096, 4097, 9000, 0, 5]


def test_group_sizes_match_fp64(gpu_ctx):
    from asz_b200 import grad
    rng = np.random.default_rng(9)
    n = np.array(SIZES * 3)
    off = np.concatenate([[0], np.cumsum(n)])
    groups, samples = len(n), int(off[-1])
    eb = rng.uniform(1e-3, 1e-2, groups).astype(np.float32)
    slope = rng.uniform(1, 30, groups).astype(np.float32)
    t = rng.uniform(0.07, 0.37, groups).astype(np.float32)
    per = lambda v: np.repeat(v.astype(np.float64), n)
    q = np.floor(rng.normal(0, 20, samples)).clip(-90, 90) + rng.uniform(0.1, 0.9, samples)
    A = rng.normal(0, 0.05, samples).astype(np.float32)
    B = (q * 2 * per(eb) - A * per(t)).astype(np.float32)
    meta = np.stack([eb, 0.2 * eb, 2.5 / eb, slope], 1).astype(np.float32)
    dev = lambda v, k: torch.tensor(v, dtype=k, device="cuda")
    info = grad.GradProblem(groups=groups, samples=samples, R2=4.0)
    a, b = dev(A, torch.float32), dev(B, torch.float32)
    prob = grad.Problem(a, b, dev(off, torch.int32), dev(meta, torch.float32), info, (a, b))
    tt = dev(t, torch.float32).requires_grad_(True)
    J = grad.RelaxedProxy.apply(tt, prob)
    J.sum().backward()
    t64 = tt.detach().double().requires_grad_(True)
    J64 = relaxed_proxy_torch(a.double(), b.double(), prob.offsets, prob.meta.double(), 4.0, t64)
    J64.sum().backward()
    # A sample's weight is off by the float roundings of q (|q| < 100, four of them) and of the
    # fixed-point weight (2^-20 at least); an entropy's term changes by log2(1 / EPS) times that.
    weight = 100 * 4 * 2.0 ** -24 + 2.0 ** -20
    bound = slope * 2 * weight * (np.log2(1 / EPS) + 1.5) + 1e-4
    got, want = J.detach().cpu().numpy(), J64.detach().cpu().numpy()
    assert (np.abs(got - want) <= bound).all(), np.abs(got - want).max()
    assert (got[n == 0] == 0).all() and (tt.grad.cpu().numpy()[n == 0] == 0).all()
    # h' of a bin holding at least a tenth of a sample: d log2(p) = weight / p, so the difference of
    # two of them is off by at most 2 * 3 * weight / (0.1 / n) / n per sample, at |dq/dt| = |A| / 2eb.
    mean_dq = np.array([np.abs(A[off[i]:off[i + 1]]).mean() / (2 * eb[i]) if n[i] else 0.0 for i in range(groups)])
    gb = slope * mean_dq * 6 * weight / 0.1 + 1e-4 * (1 + np.abs(t64.grad.cpu().numpy()))
    err = np.abs(tt.grad.cpu().numpy() - t64.grad.cpu().numpy())
    assert (err <= gb).all(), (err / gb).max()
