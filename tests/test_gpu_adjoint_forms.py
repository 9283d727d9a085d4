"""The adjoint's two replays -- fixed-point table with ratio derivative tables, and the exact blend with
linear ones (tables with steep bins) -- over the shapes of 4, 8, 16 and 32 lanes, full and
padded, and pass lengths that leave partial groups of steps, against the FP64 form's central differences in
mu_s and sigma. Needs a B200.

Both sides see the same proposals; the difference quotient's own error at h = 1e-3 relative and the
FP32 replay's agree to 1e-3, the tolerance of the single-configuration checks."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu
H = 1e-3


def _run(N, mu_s, sigma, form, steps):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.55 * S, 0.1 * S, 0), (1, 0, 0), S)
    eps = float(np.float32(sigma * sigma))
    p = T.default_params(num_segments=N, mu=1.0, eps=eps, scatter=float(mu_s), num_steps_int=2000, num_curvature_steps=2048,
                         form=form, lut_mode=T.LUT_FP64, perturb_seed=3, num_chains=700, paths_to_generate=700 * steps,
                         paths_to_skip=30, max_sub_chain=32, max_angle=0.05)
    return p, bc


@pytest.mark.parametrize("sigma", [0.1, 0.2])
@pytest.mark.parametrize("N,steps", [(10, 33), (16, 5), (34, 17), (64, 9), (130, 33), (200, 7), (256, 16), (514, 5), (701, 33)])
def test_adjoint_matches_fp64_differences(N, steps, sigma):
    p, bc = _run(N, 10.0, sigma, T.FORM_COMPENSATED, steps)
    with T.Context(p) as ctx:
        fwd = ctx.run(bc)
        g = ctx.adjoint(bc, fwd)

    def log10w(mu_s, sg):
        q, b = _run(N, mu_s, sg, T.FORM_FP64, steps)
        with T.Context(q) as ctx:
            return ctx.run(b).log10_weight, float(np.sqrt(np.float64(q.eps))), float(q.scatter)

    hi, lo = log10w(10.0 * (1 + H), sigma), log10w(10.0 * (1 - H), sigma)
    d_mu = (hi[0] - lo[0]) / (hi[2] - lo[2])
    hi, lo = log10w(10.0, sigma * (1 + H)), log10w(10.0, sigma * (1 - H))
    d_sigma = (hi[0] - lo[0]) / (hi[1] - lo[1])
    assert abs(g[0] - d_mu) < 1e-3 * abs(d_mu)
    assert abs(g[1] - d_sigma) < 1e-3 * abs(d_sigma)
    assert np.all(np.isfinite(g))


@pytest.mark.parametrize("N", [16, 66, 258])
def test_batched_and_single_adjoint_agree_with_and_without_steep_bins(N):
    """sigma = 0.05 gives steep bins (the exact replay), 0.15 none (the fixed-point one); a batch holds both."""
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.55 * S, 0.1 * S, 0), (1, 0, 0), S)
    kw = dict(num_segments=N, mu=1.0, scatter=10.0, num_steps_int=2000, num_curvature_steps=2048, form=T.FORM_COMPENSATED,
              lut_mode=T.LUT_FP64, perturb_seed=3, bootstrap_seed=4, num_chains=256, paths_to_generate=256 * 21, paths_to_skip=30,
              max_sub_chain=32, max_angle=0.05)
    eps = [float(np.float32(s * s)) for s in (0.05, 0.15)]
    with T.Context(T.default_params(eps=eps[0], **kw)) as ctx:
        res, grad, _, _ = ctx.adjoint_batch([T.make_experiment(bc, N, 10.0, e, 256 * 21) for e in eps])
    assert res[0].steep_bins > 0 and res[1].steep_bins == 0
    for i, e in enumerate(eps):
        with T.Context(T.default_params(eps=e, experiment_id=i, **dict(kw, bootstrap_seed=4 + i))) as ctx:
            fwd = ctx.run(bc)
            g = ctx.adjoint(bc, fwd)
        assert np.all(np.abs(grad[i] - g) < 1e-5 * np.max(np.abs(g[2:])) + 1e-5 * np.abs(g))
