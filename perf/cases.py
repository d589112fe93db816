"""The work that users of the framework have it do, as cases of one pass each.

The framework is an error-bounded compressor for 3-D float32 fields, and what its users call is
small in number: compress a field (one call, many fields in one call, with the plan given or
searched for), decompress a stream, tune the per-block coefficients by gradient and compress with
them, differentiate the tuner's proxy, sweep the predictors over a field, and check a
reconstruction. A case names one of these ("do") and its sizes, data and options; the fields are
seeded Gaussian random fields of the spectra and fronts of the benchmark workloads, made on the GPU.

A program keeps one `Context` for all its fields, so this module keeps one too. Streams go, whole,
into the buffer that such a program writes its archive from (their length beside them),
reconstructions come back as whole arrays.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from asz_b200 import api, grad, sweep

#: Longest pass of a drawn case, as values of the field.
MOST_VALUES = 1 << 26

_CONTEXT = None


def _context():
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = api.Context(0)
    return _CONTEXT


def listed():
    return [
        # One small block of a simulation, compressed where it lies: the call's launches and waits.
        dict(name="compress_small", do="compress", d0=40, d1=48, d2=64, eb=1e-3, family="cubic", plan="axis2",
             layers=5, bpr=3, alpha=5 / 3, front=True, host=False),
        # What s1_compress does by default with a raw file in host memory: plan search and family
        # selection on, launcher's block ratio (the 100x500x500 weather-like field).
        dict(name="compress_auto", do="compress", d0=100, d1=500, d2=500, eb=1e-3, family="auto", plan="auto",
             layers=0, bpr=3, alpha=11 / 3, front=False, host=True),
        # The throughput workload: a large field on the GPU with a reused plan.
        dict(name="compress_512", do="compress", d0=512, d1=512, d2=512, eb=1e-3, family="cubic", plan="axis2",
             layers=9, bpr=3, alpha=5 / 3, front=True, host=False),
        # A ragged field at a tight bound with a plan over all axes, quintic.
        dict(name="compress_ragged", do="compress", d0=161, d1=257, d2=349, eb=1e-4, family="quintic", plan="mixed",
             layers=9, bpr=4, alpha=3.0, front=False, host=False),
        # Reading a small stream back into host memory.
        dict(name="decompress_small", do="decompress", d0=40, d1=48, d2=64, eb=1e-3, family="cubic", plan="axis2",
             layers=5, bpr=3, alpha=5 / 3, front=True, host=True),
        # Reading a large stream back onto the GPU, for analysis there.
        dict(name="decompress_512", do="decompress", d0=512, d1=512, d2=512, eb=1e-3, family="cubic", plan="axis2",
             layers=9, bpr=3, alpha=5 / 3, front=True, host=False),
        # The same for a ragged field written with a plan over all axes at a tight bound.
        dict(name="decompress_ragged", do="decompress", d0=161, d1=257, d2=349, eb=1e-4, family="quintic",
             plan="mixed", layers=9, bpr=4, alpha=3.0, front=False, host=False),
        # Several variables of one snapshot, uneven shapes, one call with one plan.
        dict(name="batch", do="batch", count=8, lo=96, hi=256, shapes=3, eb=1e-3, family="cubic", plan="mixed",
             layers=9, bpr=3, alpha=4.0),
        # A time step with a reused plan: samples gathered, coefficients tuned by gradient, stream written.
        dict(name="tuned", do="tuned", d0=256, d1=256, d2=256, eb=1e-3, family="cubic", plan="mixed", layers=9, bpr=3,
             alpha=3.5, front=True),
        # A caller's own optimiser on the tuner's proxy: forward and backward over every group.
        dict(name="proxy", do="proxy", d0=256, d1=256, d2=256, eb=1e-3, plan="mixed", layers=9, bpr=3, alpha=3.5,
             front=True),
        # The study tool: one predictor over its coefficient grid.
        dict(name="sweep", do="sweep", d0=100, d1=500, d2=500, eb=1e-3, predictor="1d4r2_xx2", targets="legacy",
             grid="legacy", alpha=11 / 3),
        # The check after a round trip: largest error and PSNR of a reconstruction on the GPU.
        dict(name="verify", do="verify", d0=256, d1=256, d2=256, eb=1e-3, alpha=5 / 3),
    ]


def draw(rng):
    do = rng.choice(["compress", "compress", "compress", "decompress", "decompress", "batch", "tuned", "proxy",
                     "sweep", "verify"])
    alpha = round(rng.uniform(1.6, 5.0), 2)
    eb = float("%.2g" % 10 ** rng.uniform(-5, -2))
    bpr = rng.choice([3, 4])
    if do == "batch":
        return dict(do=do, count=rng.randint(2, 12), lo=rng.randint(48, 128), hi=rng.randint(129, 224),
                    shapes=rng.randint(0, 999), eb=eb, family=rng.choice(["cubic", "quintic"]),
                    plan=rng.choice(["axis2", "mixed"]), layers=rng.choice([6, 9]), bpr=bpr, alpha=alpha)
    most = MOST_VALUES if do in ("compress", "decompress", "verify") else MOST_VALUES // 4
    values = math.exp(rng.uniform(math.log(2e4), math.log(most)))
    side = values ** (1 / 3)
    d0 = max(16, round(side * math.exp(rng.uniform(-0.6, 0.6))))
    d1 = max(16, round(side * math.exp(rng.uniform(-0.6, 0.6))))
    d2 = max(16, int(values / (d0 * d1)))
    case = dict(do=do, d0=d0, d1=d1, d2=d2, eb=eb, alpha=alpha)
    if do == "verify":
        return case
    if do == "sweep":
        return dict(case, predictor=rng.choice(sweep.predictors("all")), targets=rng.choice(["legacy", "common"]),
                    grid="legacy")
    plan = rng.choice(["axis2", "mixed", "mixed"])
    # As many rounds as the smallest of the plan's axes has strides for.
    deep = int(math.log2(min(d0, d1, d2) if plan == "mixed" else d2)) - 1
    case.update(plan=plan, layers=min(9, 3 * max(1, deep) if plan == "mixed" else deep), bpr=bpr,
                front=rng.random() < 0.5)
    if do == "proxy":
        return case
    case["family"] = rng.choice(["cubic", "quintic"])
    if do == "compress" and rng.random() < 0.25:
        case.update(plan="auto", layers=0, family="auto")
    if do != "tuned":
        case["host"] = rng.random() < 0.4
    return case


def _plan(case):
    """axis2: every round along the last axis; mixed: the axes in turn; auto: searched for."""
    if case["plan"] == "auto":
        return None
    if case["plan"] == "axis2":
        return ",".join(["cubic2_012"] * case["layers"])
    turn = ["cubic0_012", "cubic1_120", "cubic2_012"]
    return ",".join(turn[i % 3] for i in range(case["layers"]))


def _params(case):
    return api.default_params(block_pivot_ratio=case["bpr"])


def _shape(case):
    return case["d0"], case["d1"], case["d2"]


def _field(shape, alpha, front, seed):
    """A Gaussian random field with P(k) ~ k^-alpha and unit variance, plus a tanh front of width 4
    and ten times its deviation, or white noise at 1e-4 of the range."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    spec = torch.fft.rfftn(torch.randn(shape, generator=g, device="cuda"))
    k = [torch.fft.fftfreq(n, device="cuda") * n for n in shape[:-1]]
    k.append(torch.fft.rfftfreq(shape[-1], device="cuda") * shape[-1])
    kk = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    kk[0, 0, 0] = 1.0
    amp = kk.pow_(-alpha / 4.0)
    amp[0, 0, 0] = 0.0
    f = torch.fft.irfftn(spec.mul_(amp), s=shape)
    f -= f.mean()
    f /= f.std()
    if front:
        gen = np.random.default_rng(seed)
        nrm = gen.standard_normal(3)
        nrm /= np.linalg.norm(nrm)
        c = [gen.uniform(0.25 * n, 0.75 * n) for n in shape]
        ax = [torch.arange(n, device="cuda", dtype=torch.float32) for n in shape]
        d = (ax[0][:, None, None] - c[0]) * nrm[0] + (ax[1][None, :, None] - c[1]) * nrm[1]
        f += 10.0 * torch.tanh((d + (ax[2][None, None, :] - c[2]) * nrm[2]) / 4.0)
    else:
        f += torch.randn(shape, generator=g, device="cuda") * (1e-4 * float(f.max() - f.min()))
    return f.contiguous()


def prepare(case, seed):
    do, ctx = case["do"], _context()
    state = dict(do=do, ctx=ctx, case=case)
    if do == "batch":
        rng = np.random.default_rng(case["shapes"])
        shapes = [tuple(int(v) for v in rng.integers(case["lo"], case["hi"] + 1, size=3)) for _ in range(case["count"])]
        state["fields"] = [_field(s, case["alpha"], False, 1000 * seed + i) for i, s in enumerate(shapes)]
        state["plan"], state["params"] = _plan(case), _params(case)
        state["archive"] = [_archive(case, math.prod(s)) for s in shapes]
        return state
    if do == "sweep":
        state["x"] = _field(_shape(case), case["alpha"], False, seed)
        return state
    if do == "verify":
        x = _field(_shape(case), case["alpha"], False, seed)
        span = float(x.max() - x.min())
        step = 2 * case["eb"] * span
        state.update(x=x, y=torch.round(x / step) * step, span=span)
        return state
    x = _field(_shape(case), case["alpha"], case["front"], seed)
    plan, p = _plan(case), _params(case)
    state.update(plan=plan, params=p)
    torch.cuda.synchronize()  # the field is there before the context's own stream reads it
    if do == "compress":
        state["x"] = x.cpu().numpy() if case["host"] else x
        state["archive"] = [_archive(case, x.numel())]
    elif do == "decompress":
        state["blob"] = ctx.compress(x, case["eb"], plan, case["family"], p)[0]
        state["out"] = None if case["host"] else torch.empty_like(x)
    elif do == "tuned":
        state["x"] = x
        state["archive"] = [_archive(case, x.numel())]
    elif do == "proxy":
        state["problem"] = grad.prepare(ctx, x, case["eb"], plan, p)
        g = torch.Generator(device="cuda").manual_seed(seed)
        lo, hi = state["problem"].info.t_min, state["problem"].info.t_max
        state["t"] = lo + (hi - lo) * torch.rand(state["problem"].groups, generator=g, device="cuda")
    torch.cuda.synchronize()
    return state


def _stream_bytes(case, values):
    """About the bytes of a stream: 6.5 bits a value at 1e-3, one more for each halving of the bound."""
    return values * max(1.0, 6.5 + math.log2(1e-3 / case["eb"])) / 8


def _archive(case, values):
    return np.zeros(65536 + 2 * int(_stream_bytes(case, values)), dtype=np.uint8)


def _written(archive, blob):
    """The archive with the stream at its front, and the stream's length."""
    archive[: len(blob)] = np.frombuffer(blob, dtype=np.uint8)
    return {"stream": archive, "length": len(blob)}


def run(state):
    do, ctx, case = state["do"], state["ctx"], state["case"]
    if do == "compress":
        blob, _ = ctx.compress(state["x"], case["eb"], state["plan"], case["family"], state["params"])
        return _written(state["archive"][0], blob)
    if do == "decompress":
        return ctx.decompress(state["blob"], _shape(case), case["eb"], state["params"], state["out"])[0]
    if do == "batch":
        blobs, _, _ = ctx.compress_batch(state["fields"], case["eb"], state["plan"], case["family"], state["params"])
        return [_written(a, b) for a, b in zip(state["archive"], blobs)]
    if do == "tuned":
        problem = grad.prepare(ctx, state["x"], case["eb"], state["plan"], state["params"])
        codes, _ = grad.tune(problem)
        blob, _ = ctx.compress_with_t(state["x"], case["eb"], state["plan"], case["family"], state["params"], codes)
        return {"codes": codes, **_written(state["archive"][0], blob)}
    if do == "proxy":
        t = state["t"].clone().requires_grad_(True)
        score = grad.RelaxedProxy.apply(t, state["problem"])
        score.sum().backward()
        return {"score": score.detach(), "grad": t.grad}
    if do == "sweep":
        rows, span = sweep.run(ctx, state["x"], case["predictor"], [case["eb"]], case["targets"], case["grid"])
        return {"counts": np.array([[r.samples, r.huffman_bytes, r.zstd_bytes] for r in rows], dtype=np.int64),
                "figures": np.array([[r.br, r.cr, r.h1, r.rmse, r.mae, r.psnr] for r in rows], dtype=np.float64),
                "range": np.array(span, dtype=np.float32)}
    return dict(zip(("max_err", "psnr"), api.error_stats_noalloc(state["x"], state["y"], state["span"])))


def _values(case):
    if case["do"] == "batch":
        rng = np.random.default_rng(case["shapes"])
        return sum(int(np.prod(rng.integers(case["lo"], case["hi"] + 1, size=3))) for _ in range(case["count"]))
    return case["d0"] * case["d1"] * case["d2"]


def work(case):
    """The field read (or written) once and the stream written (or read) once."""
    n, do = _values(case), case["do"]
    if do == "verify":
        return {"bytes": 8 * n, "flops": 4 * n}
    if do == "sweep":
        k = len(sweep.coefficients(case["predictor"], case["grid"]))
        return {"bytes": 4 * n, "flops": 12 * n // 2 * k}
    if do == "proxy":
        # About 512 samples (two values each) of each block's round, read forward and backward.
        rounds = case["layers"]
        halved = [0, 0, rounds] if case["plan"] == "axis2" else [(rounds + 2 - a) // 3 for a in range(3)]
        blocks = math.prod(-(-d // (case["bpr"] << h)) for d, h in zip(_shape(case), halved))
        samples = min(512 * blocks * rounds, 2 * n)
        return {"bytes": 2 * 8 * samples, "flops": 2 * 20 * samples}
    return {"bytes": 4 * n + _stream_bytes(case, n), "flops": (12 if do == "decompress" else 30) * n}


def _proxy64(a, b, seg, count, eb, slope, r2, t):
    """The relaxed proxy of every group in plain torch."""
    half, bins = grad.HALF_BINS, grad.BINS
    r = a * t[seg] + b
    q = (r / (2 * eb[seg])).clamp(-half, half)
    low = torch.floor(q.detach()).clamp(max=half - 1)
    frac = q - low
    at = seg * bins + (low + half).to(torch.int64)
    w = torch.zeros(count.numel() * bins, dtype=a.dtype, device=a.device)
    w = w.index_add(0, at, 1 - frac).index_add(0, at + 1, frac)
    n = count.clamp(min=1).to(a.dtype)
    p = w.view(-1, bins) / n[:, None]
    entropy = -(p * torch.log2(p + 1e-6)).sum(1)
    m = torch.zeros_like(n).index_add(0, seg, r * r) / n
    c = eb * eb / 3
    mse = (m * c / (m + c)).clamp(min=1e-300)
    score = slope * entropy - 10 * torch.log10(r2 / mse)
    return torch.where(count > 0, score, torch.zeros_like(score))


def exact(case, seed):
    if case["do"] == "verify":
        state = prepare(case, seed)
        x, y = state["x"].double(), state["y"].double()
        mse = ((x - y) ** 2).mean().item()
        return {"max_err": float((x - y).abs().max()), "psnr": 10 * math.log10(state["span"] ** 2 / mse)}
    if case["do"] == "proxy":
        state = prepare(case, seed)
        q = state["problem"]
        count = q.offsets.to(torch.int64).diff()
        seg = torch.repeat_interleave(torch.arange(count.numel(), device=count.device), count)
        eb, slope = q.meta[:, 0].double(), q.meta[:, 3].double()
        slope = torch.where(torch.isfinite(slope), slope, torch.zeros_like(slope))
        t = state["t"].double().requires_grad_(True)
        score = _proxy64(q.A.double(), q.B.double(), seg, count, eb, slope, float(q.info.R2), t)
        score.sum().backward()
        return {"score": score.detach(), "grad": t.grad}
    # Streams and reconstructions are defined bit by bit and have no value in 64 bits.
    return None
