"""The framework's work as its users run it, case by case, through its public entry points.

A case is one call (or the short sequence of calls a program always makes together): single
experiments of every form, the differentiation form, batches of receivers, the image gradient,
the independent-sample estimator, path export and re-weighing. `listed` names the cases,
`draw` gives more of the same ranges, `prepare` builds what a program holds before the call,
`run` makes the call, `work` counts what it cannot do without and `exact` restates the result in
64 bits with torch alone.
"""
import math

import numpy as np
import torch

import twisty_b200 as T
from twisty_b200 import drivers
from twisty_b200.autograd import experiment_log10_weight

PI = float(np.float32(math.pi))
LN10 = math.log(10.0)


# ------------------------------------------------------------------------------------ cases
def _experiment(name, N, paths, bins, steps_int, skip, S, end, form=T.FORM_COMPENSATED, chains=0, k=32, angle=0.1,
                eps=0.01, scatter=10.0, absorption=0.0, **more):
    c = dict(name=name, kind="experiment", form=form, N=N, paths=paths, chains=chains, bins=bins, steps_int=steps_int,
             skip=skip, S=S, ex=end[0], ey=end[1], ez=end[2], k=k, angle=angle, eps=eps, scatter=scatter,
             absorption=absorption)
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: a short-chain experiment at the reference's proposal ranges, where
        # setup, launches and read-backs are what a caller waits for
        _experiment("experiment_smallest", 16, 1 << 14, 1024, 2000, 64, 6.0, (2.5, 1.0, 0.5), k=25, angle=PI,
                    eps=0.0025, scatter=50.0),
        # the plain method's configuration run in the default form: one ordinary experiment
        _experiment("experiment_ordinary", 64, 1 << 20, 4096, 4000, 64, 10.0, (8.0, 0.0, 0.0), chains=4096),
        # a reference-style configuration: N = 2^k + 2 from the recursive bootstrapper, a 20000-bin
        # table, sub-chains of up to 25 turned by up to pi, a long burn-in
        _experiment("experiment_reference_config", 66, 1 << 22, 20000, 2000, 1000, 10.0, (8.0, 0.0, 0.0), k=25,
                    angle=PI, absorption=0.05),
        # the precision form's configuration: the largest single experiment
        _experiment("experiment_precision", 256, 1 << 26, 8192, 20000, 256, 20.0, (0.0, 0.0, 12.0), angle=0.05),
        # a long chain of odd length
        _experiment("experiment_long", 701, 1 << 20, 4096, 4000, 128, 40.0, (0.0, 0.0, 24.0), angle=0.05),
        # the drop-in form with the reference's own arithmetic
        _experiment("experiment_plain_form", 64, 1 << 20, 4096, 4000, 64, 10.0, (8.0, 0.0, 0.0),
                    form=T.FORM_PLAIN_FP32, chains=16384),
        # the differentiation form: forward and backward through the autograd binding
        dict(name="differentiation", kind="autograd", N=128, paths=1 << 22, chains=4096, bins=4096, steps_int=4000,
             skip=2000, S=16.0, ex=8.0, k=32, angle=0.1, sigma=0.1, scatter=10.0),
        # receiver loop: uneven experiments in one call
        dict(name="batch_uneven", kind="batch", n=512, n_lo=16, n_hi=1024, paths=1 << 14, bins=4096, steps_int=2000,
             skip=64, k=32, angle=0.05),
        # image gradient: pixels of one plane, shared phase parameters, tables of a multi-arclength set
        dict(name="image_gradient", kind="image", nx=8, ny=6, N=512, paths=1 << 17, bins=4096, steps_int=2000,
             n_ds=32, skip=64, k=32, angle=0.05, sigma=0.15, scatter=20.0),
        # independent samples of the recursive bootstrapper
        dict(name="msegment", kind="msegment", N=66, paths=1 << 21, bins=8192, steps_int=4000, S=20.0, ez=12.0,
             form=T.FORM_COMPENSATED),
        # re-weighing a batch of paths that the program holds in host memory
        dict(name="reweigh", kind="reweigh", N=256, paths=1 << 14, bins=8192, steps_int=4000, S=20.0, ez=12.0,
             form=T.FORM_COMPENSATED),
        # export of an experiment's first weighted paths into the program's arrays
        dict(name="export", kind="export", N=128, paths=1 << 20, chains=2048, max_paths=3000, bins=4096,
             steps_int=4000, skip=64, S=16.0, ex=8.0, k=32, angle=0.1, form=T.FORM_COMPENSATED),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["experiment"] * 5 + ["plain", "autograd", "batch", "image", "msegment", "reweigh", "export"])
    bins = rng.choice([512, 1024, 1777, 2048, 4096, 5001, 8192, 20000])
    steps_int = rng.choice([2000, 4000, 20000])
    small = rng.random() < 0.7
    angle = rng.choice([0.05, 0.1]) if small else PI
    k = 32 if small else 25
    if kind == "experiment":
        N = _log_int(rng, 8, 1024)
        paths = _log_int(rng, 1 << 13, min(1 << 26, (1 << 33) // N))
        S = rng.uniform(8.0, 24.0)
        return dict(kind=kind, form=T.FORM_COMPENSATED, N=N, paths=paths, chains=0, bins=bins, steps_int=steps_int,
                    skip=rng.choice([0, 64, 256, 1000]), S=S, ex=0.6 * S * rng.uniform(0.5, 1.0),
                    ey=rng.uniform(-0.5, 0.5), ez=rng.uniform(-0.5, 0.5), k=k, angle=angle,
                    eps=rng.uniform(0.05, 0.3) ** 2, scatter=rng.uniform(5.0, 50.0), absorption=rng.choice([0.0, 0.05]))
    if kind == "plain":
        N = _log_int(rng, 8, 512)
        return dict(kind="experiment", form=T.FORM_PLAIN_FP32, N=N, paths=_log_int(rng, 1 << 14, (1 << 28) // N),
                    chains=rng.choice([0, 4096, 10007]), bins=bins, steps_int=steps_int, skip=rng.choice([0, 64, 200]),
                    S=10.0, ex=6.0 * rng.uniform(0.6, 1.2), ey=0.0, ez=0.3, k=k, angle=angle, eps=0.01,
                    scatter=rng.uniform(5.0, 50.0), absorption=0.0)
    if kind == "autograd":
        N = _log_int(rng, 20, 600)
        S = rng.uniform(12.0, 20.0)
        return dict(kind=kind, N=N, paths=_log_int(rng, 1 << 17, (1 << 29) // N), chains=rng.choice([1024, 4096]),
                    bins=rng.choice([1024, 2048, 4096, 5001]), steps_int=rng.choice([2000, 4000]),
                    skip=rng.choice([200, 2000]), S=S, ex=0.5 * S, k=32, angle=0.1, sigma=rng.uniform(0.08, 0.2),
                    scatter=rng.uniform(5.0, 20.0))
    if kind == "batch":
        n = _log_int(rng, 8, 1024)
        return dict(kind=kind, n=n, n_lo=16, n_hi=rng.choice([200, 1024]), paths=_log_int(rng, 1 << 10, (1 << 23) // n),
                    bins=rng.choice([1024, 2048, 4096]), steps_int=2000, skip=rng.choice([0, 64]), k=32, angle=angle)
    if kind == "image":
        nx, ny = rng.randint(2, 12), rng.randint(2, 12)
        N = _log_int(rng, 32, 700)
        return dict(kind=kind, nx=nx, ny=ny, N=N, paths=_log_int(rng, 1 << 13, (1 << 32) // (N * nx * ny)),
                    bins=rng.choice([1024, 2048, 4096]), steps_int=2000, n_ds=rng.choice([8, 32]),
                    skip=rng.choice([0, 64]), k=32, angle=0.05, sigma=rng.uniform(0.1, 0.2),
                    scatter=rng.uniform(10.0, 30.0))
    form = rng.choice([T.FORM_COMPENSATED, T.FORM_COMPENSATED, T.FORM_PLAIN_FP32])
    if kind == "msegment":
        N = rng.choice([10, 18, 34, 50, 66, 130, 258])
        return dict(kind=kind, N=N, paths=_log_int(rng, 1 << 14, (1 << 28) // N), bins=bins, steps_int=2000, S=20.0,
                    ez=rng.uniform(8.0, 14.0), form=form)
    if kind == "reweigh":
        N = _log_int(rng, 8, 1000)
        return dict(kind=kind, N=N, paths=_log_int(rng, 256, (1 << 23) // N), bins=bins, steps_int=2000, S=20.0,
                    ez=rng.uniform(8.0, 14.0), form=form)
    N = _log_int(rng, 16, 300)
    return dict(kind=kind, N=N, paths=_log_int(rng, 1 << 17, 1 << 20), chains=rng.choice([512, 2048]),
                max_paths=_log_int(rng, 100, (1 << 20) // N), bins=rng.choice([1024, 4096]), steps_int=2000, skip=64,
                S=16.0, ex=rng.uniform(6.0, 10.0), k=k, angle=angle, form=form)


# ---------------------------------------------------------------------------------- prepare
def _jitter(seed, n):
    """n offsets in [-0.02, 0.02] and two seeds: the program's own inputs differ from run to run."""
    r = np.random.default_rng(seed)
    return r.uniform(-0.02, 0.02, n), int(r.integers(1, 1 << 31)), int(r.integers(1, 1 << 31))


def _params(c, seed, **more):
    _, perturb, boot = _jitter(seed, 3)
    kw = dict(num_segments=c.get("N", 16), mu=1.0, eps=c["eps"] if "eps" in c else c.get("sigma", 0.1) ** 2,
              scatter=c.get("scatter", 10.0), absorption=c.get("absorption", 0.0), num_steps_int=c["steps_int"],
              num_curvature_steps=c["bins"], form=c.get("form", T.FORM_COMPENSATED), lut_mode=T.LUT_FP64,
              paths_to_generate=c.get("paths", 0), paths_to_skip=c.get("skip", 0), num_chains=c.get("chains", 0),
              max_sub_chain=c.get("k", 25), max_angle=c.get("angle", PI), perturb_seed=perturb, bootstrap_seed=boot)
    kw.update(more)
    return T.default_params(**kw)


def _ends(c, seed):
    """(start, start tangent, end, end tangent): along x where the receiver is, else along z."""
    off, _, _ = _jitter(seed, 3)
    e = np.array([c.get("ex", 0.0), c.get("ey", 0.0), c.get("ez", 0.0)])
    d = (1.0, 0.0, 0.0) if abs(e[0]) >= abs(e[2]) else (0.0, 0.0, 1.0)
    return (0.0, 0.0, 0.0), d, tuple(float(v) for v in np.float32(e + off)), d


def _bc(c, seed):
    return T.make_bc(*_ends(c, seed), c["S"])


def _batch(c, seed):
    """Receivers on spheres around the source, tangents anywhere, uneven N, arclength and phase."""
    r = np.random.default_rng(seed)
    out = []
    while len(out) < c["n"]:
        N = int(round(math.exp(r.uniform(math.log(c["n_lo"]), math.log(c["n_hi"])))))
        rad, d, t = r.uniform(2.0, 10.0), r.normal(size=3), r.normal(size=3)
        d, t = d / np.linalg.norm(d), t / np.linalg.norm(t)
        S, sigma, mus = rad * r.uniform(1.05, 2.0), r.uniform(0.05, 0.3), r.uniform(5.0, 50.0)
        bc = T.make_bc((0.0, 0.0, 0.0), (0.0, 0.0, 1.0), rad * d, t, S)
        if T.min_arclength(bc, N) < S:
            out.append(T.make_experiment(bc, N, mus, sigma * sigma, c["paths"]))
    return out


def _walks(c, seed):
    """Paths of N segments of length S/N whose tangents wander by about 0.1 rad a step (float32, host)."""
    g = torch.Generator().manual_seed(int(seed))
    P, N = c["paths"], c["N"]
    t = torch.zeros(P, N, 3)
    t[:, :, 2] = 1.0
    t = t + 0.1 * torch.cumsum(torch.randn(P, N, 3, generator=g), dim=1)
    t = t / t.norm(dim=2, keepdim=True)
    pos = torch.zeros(P, N + 1, 3)
    pos[:, 1:] = torch.cumsum(t * (c["S"] / N), dim=1)
    return pos.numpy()


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "experiment":
        _, perturb, boot = _jitter(seed, 3)
        w = T.WeightingParameters(mu=1.0, numStepsInt=c["steps_int"], maxBound=float(np.float32(10.0) / np.float32(c["eps"])),
                                  eps=c["eps"], scatter=c["scatter"], absorption=c["absorption"],
                                  numCurvatureSteps=c["bins"])
        p = T.ExperimentParameters(numPathsInExperiment=c["paths"], numPathsToSkip=c["skip"], numSegmentsPerCurve=c["N"],
                                   bootstrapSeed=boot, curvePurturbSeed=perturb, weightingParameters=w, form=c["form"],
                                   maxSubChain=c["k"], maxAngle=c["angle"], numChains=c["chains"])
        s, sd, e, ed = _ends(c, seed)
        return dict(kind=kind, runner=T.FullExperimentRunnerOptimalPerturbOptimized_GPU(p),
                    bc=T.BoundaryConditions(s, sd, e, ed, c["S"]))
    if kind == "autograd":
        bc = _bc(c, seed)
        leaf = lambda v: torch.tensor(v, dtype=torch.float32, requires_grad=True)  # noqa: E731
        return dict(kind=kind, params=_params(c, seed), bc=bc, mu_s=leaf(c["scatter"]), sigma=leaf(c["sigma"]),
                    receiver=leaf([bc.end_pos.x, bc.end_pos.y, bc.end_pos.z]))
    if kind == "batch":
        return dict(kind=kind, ctx=T.Context(_params(c, seed, paths_to_generate=0)), experiments=_batch(c, seed))
    if kind == "image":
        off, _, _ = _jitter(seed, 1)
        px = drivers.image_plane_experiments(c["nx"], c["ny"], 4.0, 10.0 + float(off[0]), c["N"], c["scatter"],
                                             float(np.float32(c["sigma"] ** 2)), c["paths"])
        ctx = T.Context(_params(c, seed, eps=float(np.float32(c["sigma"] ** 2)), lut_mode=T.LUT_MULTI_DS,
                                paths_to_generate=0))
        ds = [x.bc.arclength / c["N"] for x in px]
        ctx.multi_ds_tables(0.999 * min(ds), 1.001 * max(ds), c["n_ds"])
        return dict(kind=kind, ctx=ctx, experiments=px)
    ctx, bc = T.Context(_params(c, seed)), _bc(c, seed)
    if kind == "reweigh":
        return dict(kind=kind, ctx=ctx, bc=bc, pos=_walks(c, seed), form=c["form"])
    return dict(kind=kind, ctx=ctx, bc=bc, max_paths=c.get("max_paths", 0))


# -------------------------------------------------------------------------------------- run
def run(state):
    s, kind = state, state["kind"]
    if kind == "experiment":
        r = s["runner"].RunExperiment(s["bc"])
        return dict(log10_weight=r.experimentWeightLog10, log10_normalizer=r.normalizerLog10,
                    rel_std_error=r.relStdError, paths=r.totalPathsGenerated, failed=r.numFailedPaths,
                    clamped=r.clampedCurvatures)
    if kind == "autograd":
        leaves = (s["mu_s"], s["sigma"], s["receiver"])
        y = experiment_log10_weight(*leaves, s["params"], s["bc"])
        g = torch.autograd.grad(y, leaves)
        return dict(log10_weight=y.detach(), d_mu_s=g[0], d_sigma=g[1], d_receiver=g[2])
    if kind == "batch":
        return _image(s["ctx"].run_batch(s["experiments"]))
    if kind == "image":
        res, grad, total, _ = s["ctx"].adjoint_batch(s["experiments"])
        out = _image(res)
        out.update(grad=torch.from_numpy(grad).float(), total=torch.from_numpy(total).float())
        return out
    if kind == "msegment":
        r = s["ctx"].run_msegment(s["bc"])
        return dict(log10_mean_weight=r.log10_mean_weight, rel_std_error=r.rel_std_error, paths=int(r.total_paths),
                    failed=int(r.failed_paths))
    if kind == "reweigh":
        w, v, _ = s["ctx"].weight_paths(s["bc"], s["pos"], form=s["form"])
        return dict(log10_weight=w, valid=v)
    pos, w, r = s["ctx"].export_paths(s["bc"], None, s["max_paths"])
    return dict(pos=pos, log10_path_weight=w, log10_weight=r.log10_weight, paths=int(r.total_paths))


def _image(results):
    """A receiver loop's results as the program keeps them: one float image per quantity."""
    return dict(log10_weight=torch.tensor([r.log10_weight for r in results]),
                rel_std_error=torch.tensor([r.rel_std_error for r in results]),
                paths=torch.tensor([int(r.total_paths) for r in results]),
                failed=torch.tensor([int(r.failed_paths) for r in results]))


# ------------------------------------------------------------------------------------- work
def work(case):
    """A weighted path-segment costs about 40 single-precision operations (tangent, curvature, bin,
    blend, sum and its share of the rotation), a burn-in step its rotation alone; the bytes are
    the curve, the table, the paths given or returned and the results."""
    c, kind = case, case["kind"]
    per = 40.0
    if kind == "batch":
        # the mean of a log-uniform N
        n = (c["n_hi"] - c["n_lo"]) / math.log(c["n_hi"] / c["n_lo"])
        return dict(bytes=c["n"] * (64.0 + 12 * n + 4 * c["bins"]), flops=per * c["n"] * c["paths"] * n)
    if kind == "image":
        px = c["nx"] * c["ny"]
        return dict(bytes=px * (104.0 + 12 * c["N"] + 12 * c["bins"]), flops=2 * per * px * c["paths"] * c["N"])
    segs = float(c["paths"]) * c["N"]
    if kind == "reweigh":
        return dict(bytes=12.0 * c["paths"] * (c["N"] + 1) + 9 * c["paths"] + 4 * c["bins"], flops=per * segs)
    if kind == "msegment":
        return dict(bytes=4.0 * c["bins"] + 64, flops=3 * per * segs)
    own = 12.0 * (c["N"] + 1) + 4 * c["bins"] + 64
    if kind == "export":
        return dict(bytes=own + c["max_paths"] * (12.0 * (c["N"] + 1) + 8), flops=per * segs)
    if kind == "autograd":
        return dict(bytes=own + 8 * c["bins"], flops=2 * per * segs)
    return dict(bytes=own, flops=per * segs)


# ------------------------------------------------------------------------------------ exact
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _table(c, eps, scatter, ds, derivatives=False):
    """The segment-weight table over curvature in 64 bits: Simpson's rule over [0, 10/eps] with the
    two nodes before the last left out, entries that are not positive replaced by the smallest
    positive one, and the last step of the grid 2.02/ds."""
    n, bins, dev = c["steps_int"], c["bins"], _dev()
    m, bds = float(eps), float(scatter) * ds
    maxb = 10.0 / m
    h = maxb / n
    j = torch.arange(n + 1, dtype=torch.float64, device=dev)
    p = j * h
    p[-1] = maxb
    w = torch.where(j % 2 == 1, 4.0, 2.0).double()
    w[0] = w[-1] = 1.0
    w[-3:-1] = 0.0
    em = math.exp(-2.0 / m)
    norm = math.sqrt(math.pi * m * 0.5) / (1.0 - em)
    ph = norm * torch.exp(-m * p * p * 0.5)
    e = torch.exp(bds * ph - p * p * 0.5)   # mu = 1
    keep = (w * p * e) != 0
    keep[0] = True
    p, w, e, ph = p[keep], w[keep], e[keep], ph[keep]
    step = (2.0 / ds) * 1.01 / (bins - 1)
    kds = torch.arange(bins, dtype=torch.float64, device=dev) * step * ds
    scale = h / 3.0 / (2.0 * math.pi * math.pi)
    tabs = []
    for a in kds.split(512):
        x = a[:, None] * p
        s = torch.where(a[:, None] > 0, torch.sin(x) / a[:, None].clamp_min(1e-300), p.expand_as(x))
        f = p * e * s
        rows = [(f * w).sum(1) * scale]
        if derivatives:
            sp = torch.cos(x)
            f_p = e * s + p * e * (bds * (-m * p * ph) - p) * s + p * e * sp
            f_m = f * bds * ph * ((0.5 / m - (2.0 / (m * m)) * em / (1.0 - em)) - 0.5 * p * p)
            rows += [(f * ph * w).sum(1) * scale * ds, -rows[0] / m + ((-p * f_p / m + f_m) * w).sum(1) * scale]
        tabs.append(torch.stack(rows))
    t = torch.cat(tabs, dim=1)
    lut = t[0]
    low = lut[(lut.float() >= 0)].min()
    lut = torch.where(lut.float() <= 0, low, lut)
    return (lut, step, t[1], t[2]) if derivatives else (lut, step)


def _mulhi(a, b):
    """High and low 32 bits of a 32 x 32-bit product (int64 tensors holding unsigned values)."""
    a0, a1, b0, b1 = a & 0xFFFF, a >> 16, b & 0xFFFF, b >> 16
    mid = a1 * b0 + ((a0 * b0) >> 16)
    mid2 = a0 * b1 + (mid & 0xFFFF)
    return a1 * b1 + (mid >> 16) + (mid2 >> 16), ((mid2 << 16) | ((a0 * b0) & 0xFFFF)) & 0xFFFFFFFF


def _philox(c0, c1, c2, c3, seed):
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
        h0, l0 = _mulhi(c0, torch.full_like(c0, 0xD2511F53))
        h1, l1 = _mulhi(c2, torch.full_like(c2, 0xCD9E8D57))
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
    return c0, c1, c2, c3


def _arc(c, seed):
    """The planar arc of N segments between the fixed points, its plane turned by the seed (float32)."""
    s, sd, e, ed = (np.array(v, np.float32) for v in _ends(c, seed))
    boot = _jitter(seed, 3)[2]
    N = c["N"]
    ds = np.float32(c["S"]) / np.float32(N)
    pos = np.zeros((N + 1, 3), np.float32)
    pos[0], pos[1], pos[N - 1], pos[N] = s, s + sd * ds, e - ed * ds, e
    M, a0 = N - 2, pos[1].astype(np.float64)
    C = pos[N - 1].astype(np.float64) - a0
    D = np.linalg.norm(C)
    u = C / D
    ax = 0 if abs(u[0]) <= abs(u[1]) and abs(u[0]) <= abs(u[2]) else 1 if abs(u[1]) <= abs(u[2]) else 2
    w = np.eye(3)[ax] - u[ax] * u
    w /= np.linalg.norm(w)
    z, full = boot, (1 << 64) - 1
    z = (z + 0x9E3779B97F4A7C15) & full
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & full
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & full
    z ^= z >> 31
    phi = 2.0 * math.pi * (z >> 11) * 2.0 ** -53
    w2 = math.cos(phi) * w + math.sin(phi) * np.cross(u, w)
    lo, hi, dsd = 0.0, 2.0 * math.pi / M, float(ds)
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        if dsd * math.sin(0.5 * M * mid) / math.sin(0.5 * mid) > D:
            lo = mid
        else:
            hi = mid
    beta = 0.5 * (lo + hi)
    th = -0.5 * (M - 1) * beta + np.arange(M - 1) * beta
    pos[2:N - 1 + 0] = (a0 + np.cumsum(dsd * (np.cos(th)[:, None] * u + np.sin(th)[:, None] * w2), 0))[:N - 3]
    return pos


def _layout(paths, chains):
    C = min(chains, paths)
    L = -(-paths // C)
    C = -(-paths // L)
    return C, L, paths - (C - 1) * L


def _curvature(pos, inv_ds):
    v = pos[:, 1:] - pos[:, :-1]
    t = v / v.norm(dim=2, keepdim=True)
    d = t[:, 1:] - t[:, :-1]
    return t, d, d.norm(dim=2) * inv_ds


def _bins(kappa, lut, step):
    b = (kappa / step).floor().long().clamp_(0, lut.numel() - 1)
    nxt = (b + 1).clamp_max(lut.numel() - 1)
    return b, nxt, kappa - b * step


def _chains(c, seed, visit, first=None):
    """The Markov chains of one experiment in 64 bits, all of them side by side: a step turns the
    points between two random ones about their chord; visit(step, positions, chains that weigh)."""
    dev, N = _dev(), c["N"]
    C, L, last = _layout(c["paths"], c["chains"])
    if first is not None:
        C, last = min(C, first), (last if C <= first else L)
    perturb = _jitter(seed, 3)[1]
    pos = torch.from_numpy(_arc(c, seed)).double().to(dev).expand(C, N + 1, 3).contiguous()
    chain = torch.arange(C, dtype=torch.int64, device=dev)
    exp_id, tag = torch.zeros_like(chain), torch.full_like(chain, 0x54575354)
    keff = min(c["k"], N - 2)
    at = torch.arange(keff + 1, device=dev)
    rows = chain[:, None]
    for s in range(c["skip"] + L):
        r0, r1, r2, _ = _philox(torch.full_like(chain, s), chain, exp_id, tag, perturb)
        k = 2 + ((r0 * (keff - 1)) >> 32)
        left = 1 + ((r1 * (N - k - 1)) >> 32)
        signed = torch.where(r2 >= 1 << 31, r2 - (1 << 32), r2) >> 8
        u = signed.float() * 2.0 ** -23 + 2.0 ** -24
        a = (u * torch.tensor(c["angle"], dtype=torch.float32, device=dev)).double()
        idx = (left[:, None] + at).clamp_max(N)
        win = pos[rows, idx]
        base = win[:, :1]
        axis = pos[chain, left + k] - base[:, 0]
        axis = (axis / axis.norm(dim=1, keepdim=True))[:, None]
        v = win - base
        sn, cs = torch.sin(a)[:, None, None], torch.cos(a)[:, None, None]
        ax = axis.expand_as(v)
        turned = v * cs + torch.cross(ax, v, dim=2) * sn + ax * ((ax * v).sum(2, keepdim=True) * (1 - cs)) + base
        move = ((at >= 1) & (at[None] < k[:, None]))[:, :, None]
        pos[rows, idx] = torch.where(move, turned, win)
        if s >= c["skip"]:
            w = s - c["skip"]
            visit(w, pos, (chain < C - 1) | (w < last))


def _sums(logs):
    """log10 of the summed weights and the standard error from the spread over chains."""
    m = logs.max()
    x = torch.exp((logs - m) * LN10)
    n, s1 = x.numel(), x.sum()
    var = ((x * x).sum() - s1 * s1 / n) / (n - 1)
    return float(m + torch.log10(s1)), float(torch.sqrt(n * var) / s1)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "reweigh":
        return _exact_reweigh(c, seed)
    if kind == "msegment":
        return _exact_msegment(c, seed)
    # chains from the recursive bootstrapper's curve, from a chain count the library chooses, or that
    # rounding leads apart (turns of up to pi), have no value of their own; nor have receiver loops here
    if kind not in ("experiment", "autograd", "export") or not c["chains"] or c["angle"] > 0.2 or _resolvable(c["N"]):
        return None
    C, L, _ = _layout(c["paths"], c["chains"])
    if kind != "export" and (c["skip"] + L) * max(1.0, C * c["N"] / 2e6) > 6000:
        return None
    S, N, dev = float(np.float32(c["S"])), c["N"], _dev()
    ds = float(np.float32(S) / np.float32(N))
    eps = float(np.float32(c["eps"])) if "eps" in c else float(np.float32(c.get("sigma", 0.1)) * np.float32(c.get("sigma", 0.1)))
    scatter = float(np.float32(c["scatter"] if "scatter" in c else 10.0))
    absorb = math.log10(math.exp(-float(np.float32(c.get("absorption", 0.0))) * ds)) * (N - 1)
    if kind == "autograd":
        return _exact_gradient(c, seed, N, ds, S, eps, scatter)
    lut, step = _table(c, eps, scatter, ds)
    logw = []

    def weigh(_, pos, live):
        kappa = _curvature(pos, N / S)[2]
        b, nxt, f = _bins(kappa, lut, step)
        w = torch.log10(lut[b] * (1 - f) + lut[nxt] * f).sum(1) + absorb
        logw.append(torch.where(live, w, torch.tensor(-math.inf, dtype=torch.float64, device=dev)))

    if kind == "export":
        n = min(c["max_paths"], c["paths"])
        seen = []

        def keep(_, pos, live):
            weigh(_, pos, live)
            seen.append(pos.float().cpu())   # 64-bit positions, kept in the 32 bits that they come back in

        _chains(c, seed, keep, first=-(-n // L))
        w = torch.stack(logw, 1).reshape(-1)[:n]
        return dict(pos=torch.stack(seen, 1).reshape(-1, N + 1, 3)[:n].double().numpy(), log10_path_weight=w.cpu().numpy(),
                    log10_weight=None, paths=None)
    _chains(c, seed, weigh)
    t = torch.stack(logw, 1)
    m = t.max(dim=1, keepdim=True).values
    total, se = _sums((m + torch.log10(torch.exp((t - m) * LN10).sum(1, keepdim=True)))[:, 0])
    return dict(log10_weight=torch.tensor(total, dtype=torch.float64), log10_normalizer=None,
                rel_std_error=torch.tensor(se, dtype=torch.float64), paths=None, failed=None, clamped=None)


def _exact_gradient(c, seed, N, ds, S, eps, scatter):
    """The weight-averaged path gradient: the table's derivatives in mu_s and eps, and for the receiver
    the slope of the weight averaged over a bin, which is the chord of the bin half a step below."""
    lut, step, dmu, deps = _table(c, eps, scatter, ds, derivatives=True)
    acc = []

    def visit(_, pos, live):
        t, d, kappa = _curvature(pos, N / S)
        b, nxt, f = _bins(kappa, lut, step)
        v = lut[b] + f * (lut[nxt] - lut[b])
        w = torch.log10(v).sum(1)
        gm = ((dmu[b] + f * (dmu[nxt] - dmu[b])) / v).sum(1) / LN10
        ge = ((deps[b] + f * (deps[nxt] - deps[b])) / v).sum(1) / LN10
        seg = (pos[:, N - 1] - pos[:, N - 2]).norm(dim=1, keepdim=True)
        g = torch.zeros_like(seg).expand(-1, 3)
        t2 = t[:, N - 2]
        for i, sign in ((N - 3, 1.0), (N - 2, -1.0)):
            J = (kappa[:, i] / step - 0.5).floor().long().clamp_(0, lut.numel() - 2)
            slope = (lut[J + 1] - lut[J]) / (step * v[:, i]) / LN10
            e = d[:, i]
            dk = (slope * (N / S) * sign / e.norm(dim=1))[:, None]
            g = g + dk * (e - (e * t2).sum(1, keepdim=True) * t2) / seg
        acc.append(torch.cat([torch.where(live, w, torch.tensor(-math.inf, dtype=w.dtype, device=w.device))[:, None],
                              gm[:, None], ge[:, None], g], 1))

    _chains(c, seed, visit)
    a = torch.stack(acc, 1).reshape(-1, 6)
    m = a[:, 0].max()
    x = torch.exp((a[:, 0] - m) * LN10)
    g = (x[:, None] * a[:, 1:]).sum(0) / x.sum()
    sigma = math.sqrt(eps)
    return dict(log10_weight=(m + torch.log10(x.sum())).cpu(), d_mu_s=g[0].cpu(), d_sigma=(g[1] * 2 * sigma).cpu(),
                d_receiver=g[2:].cpu())


def _exact_reweigh(c, seed):
    S, N, dev = float(np.float32(c["S"])), c["N"], _dev()
    lut, step = _table(c, float(np.float32(0.1 ** 2)), 10.0, float(np.float32(S) / np.float32(N)))
    out = []
    for pos in torch.from_numpy(_walks(c, seed)).split(4096):
        kappa = _curvature(pos.to(dev).double(), N / S)[2]
        b, nxt, f = _bins(kappa, lut, step)
        out.append(torch.log10(lut[b] * (1 - f) + lut[nxt] * f).sum(1).cpu())
    return dict(log10_weight=torch.cat(out).numpy(), valid=None)


def _resolvable(N):
    m = N - 2
    while m > 6 and m % 2 == 0:
        m //= 2
    return m in (4, 6)


class _Draws:
    """The uniform draws of many paths side by side, a counter each; `where` draws for some of them."""

    def __init__(self, n, seed, dev):
        self.path = torch.arange(n, dtype=torch.int64, device=dev)
        self.zero, self.tag = torch.zeros_like(self.path), torch.full_like(self.path, 0x4D534547)
        self.count, self.seed = torch.zeros_like(self.path), seed

    def word(self, where):
        r = _philox(self.count, self.path, self.zero, self.tag, self.seed)[0]
        self.count = self.count + where
        return r

    def single(self, where):
        return (self.word(where) >> 8).double() / 16777216.0

    def double(self, where):
        hi, lo = self.word(where), self.word(where)
        return ((hi << 21) | (lo >> 11)).double() / 9007199254740992.0


def _exact_msegment(c, seed):
    """The recursive bootstrapper over every path at once: a span's centre point is drawn in the
    intersection of two balls around its ends, a span of two closes by a turn about its chord."""
    N = c["N"]
    if N - 2 & N - 3 or c["paths"] * N > 1 << 29:
        return None
    dev, P = _dev(), c["paths"]
    S = float(np.float32(c["S"]))
    ds = float(np.float32(S) / np.float32(N))
    s, sd, e, ed = (np.array(v, np.float32) for v in _ends(c, seed))
    f = np.float32(ds)
    at = {i: torch.from_numpy(v).double().to(dev).expand(P, 3) for i, v in
          ((0, s), (1, s + f * sd), (N - 1, e - f * ed), (N, e))}
    g, failed = _Draws(P, _jitter(seed, 3)[1], dev), torch.zeros(P, dtype=torch.bool, device=dev)

    def frame(a, b):
        z = b - a
        z = z / z.norm(dim=1, keepdim=True)
        x = torch.tensor([1.0, 0, 0], dtype=torch.float64, device=dev).expand_as(z)
        y = torch.tensor([0, 1.0, 0], dtype=torch.float64, device=dev).expand_as(z)
        h = torch.where(z[:, :1].abs() > 0.999, y, x)
        xa = torch.cross(z, h, dim=1)
        xa = xa / xa.norm(dim=1, keepdim=True)
        ya = torch.cross(z, xa, dim=1)
        return xa, ya, z

    def centre(m, l, r):
        nonlocal failed
        a, b, h = at[l], at[r], m // 2
        d = (b - a).norm(dim=1)
        straight = (m * ds - d).abs() < 0.001
        rad = ds * h
        failed = failed | (~straight & (2 * rad < d))
        go = (~straight).long()
        u = g.double(go) * (0.5 - 0.25 * d / rad)
        cph = 1 - 2 * u
        sph = torch.sqrt((1 - cph * cph).clamp_min(0))
        theta = g.double(go) * (2 * math.pi)
        flip = (g.word(go) & 1) == 1
        minp = 0.5 * d / cph / rad
        sr = rad * (minp + (1 - minp) * g.single(go)) ** (1.0 / 3.0)
        xa, ya, za = frame(a, b)
        side = xa * (sph * torch.cos(theta))[:, None] + ya * (sph * torch.sin(theta))[:, None]
        z = za * cph[:, None]
        p = torch.where(flip[:, None], b + (side - z) * sr[:, None], a + (side + z) * sr[:, None])
        at[l + h] = torch.where(straight[:, None], 0.5 * (a + b), p)

    def two(l, r):
        nonlocal failed
        a, b = at[l], at[r]
        d = (b - a).norm(dim=1)
        straight = (2 * ds - d).abs() < 0.001
        failed = failed | (~straight & (2 * ds < d))
        theta = g.single((~straight).long()) * (2 * math.pi)
        axis = (b - a) / d[:, None]
        x = torch.tensor([1.0, 0, 0], dtype=torch.float64, device=dev).expand_as(axis)
        y = torch.tensor([0, 1.0, 0], dtype=torch.float64, device=dev).expand_as(axis)
        n = torch.cross(axis, torch.where(axis[:, :1].abs() >= 0.99, y, x), dim=1)
        n = n / n.norm(dim=1, keepdim=True)
        off = torch.sqrt((ds * ds - 0.25 * d * d).clamp_min(0))[:, None]
        # the reference's quaternion product turns by +theta about the axis
        n = n * torch.cos(theta)[:, None] + torch.cross(axis, n, dim=1) * torch.sin(theta)[:, None]
        at[l + 1] = torch.where(straight[:, None], 0.5 * (a + b), 0.5 * (a + b) + n * off)

    def span(m, l, r):
        centre(m, l, r)
        h = m // 2
        for a, b in ((l, l + h), (l + h, r)):
            two(a, b) if h == 2 else span(h, a, b)

    span(N - 2, 1, N - 1)
    if bool(failed.any()):
        return None
    lut, step = _table(c, float(np.float32(0.1 ** 2)), 10.0, ds)
    logs = torch.zeros(P, dtype=torch.float64, device=dev)
    prev = None
    for i in range(N):
        t = at[i + 1] - at[i]
        t = t / t.norm(dim=1, keepdim=True)
        if prev is not None:
            b, nxt, fr = _bins((t - prev).norm(dim=1) * (N / S), lut, step)
            logs += torch.log10(lut[b] * (1 - fr) + lut[nxt] * fr)
        prev = t
    total, se = _sums(logs)
    return dict(log10_mean_weight=torch.tensor(total - math.log10(P), dtype=torch.float64),
                rel_std_error=torch.tensor(se, dtype=torch.float64), paths=None, failed=None)
