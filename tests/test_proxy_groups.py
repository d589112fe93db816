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


@pytest.mark.parametrize("width", [2.0 ** -6, 2.0 ** -12, 2.0 ** -18], ids=["2^-6", "2^-12", "2^-18"])
def test_weights_of_thin_bins(gpu_ctx, width):
    """Groups of well predicted samples, all within a small part of a bin of zero on its upper side: next
    to the bin that holds them, one holds only what each weighs there. The samples' coordinates have
    no rounding in float, so what is off against 64 bits comes from the weights, their sums and what follows.
    Every other sample lies far outside the bins: the squared residual is theirs, and so the gradient the entropy's."""
    from asz_b200 import grad
    rng = np.random.default_rng(11)
    n = np.array([1, 7, 33, 511, 1500, 2047, 2048, 3000, 4095, 4096, 6000] * 2)
    off = np.concatenate([[0], np.cumsum(n)])
    groups, samples = len(n), int(off[-1])
    # eb = 1/2 and t = 1/4: q = A / 4 + B, both parts multiples of width 2^-22 below width.
    unit = width * 2.0 ** -22
    A = (rng.integers(0, 1 << 21, samples) * 4 * unit).astype(np.float32)
    B = (rng.integers(1, 1 << 21, samples) * unit).astype(np.float32)
    A[1::2], B[1::2] = 0, 1000
    slope = rng.uniform(1, 30, groups).astype(np.float32)
    meta = np.stack([np.full(groups, 0.5), np.full(groups, 0.1), np.full(groups, 5.0), slope], 1).astype(np.float32)
    dev = lambda v, k: torch.tensor(v, dtype=k, device="cuda")
    a, b = dev(A, torch.float32), dev(B, torch.float32)
    prob = grad.Problem(a, b, dev(off, torch.int32), dev(meta, torch.float32), grad.GradProblem(groups=groups, samples=samples, R2=4.0),
                        (a, b))
    tt = torch.full((groups,), 0.25, device="cuda").requires_grad_(True)
    J = grad.RelaxedProxy.apply(tt, prob)
    J.sum().backward()
    t64 = tt.detach().double().requires_grad_(True)
    J64 = relaxed_proxy_torch(a.double(), b.double(), prob.offsets, prob.meta.double(), 4.0, t64)
    J64.sum().backward()
    # h' = -(log2(p + EPS) + p / (p + EPS) / ln 2): p and p + EPS are each rounded a few times (a sum of
    # floats, 1 / n: 2^-21 of their size in all), log2 is a float of up to 20 (two units in the last place,
    # 2^-18). The gradient is the mean of h' differences times dq/dt = A, at |slope|.
    mean_dq = np.array([A[off[i]:off[i + 1]].astype(np.float64).mean() for i in range(groups)])
    g64 = t64.grad.cpu().numpy()
    bound = slope * mean_dq * 2 * (3 * 2.0 ** -21 + 2.0 ** -18) + 2.0 ** -20 * np.abs(g64)
    err = np.abs(tt.grad.cpu().numpy() - g64)
    assert (err <= bound).all(), (err / bound).max()
    bound = slope * 2 * 2.0 ** -18 + 2.0 ** -20 * np.abs(J64.detach().cpu().numpy())
    err = np.abs(J.detach().cpu().numpy() - J64.detach().cpu().numpy())
    assert (err <= bound).all(), (err / bound).max()
