"""The batched adjoint over a multi-arclength table set, with experiments that share a table and differ in the replay
it takes: below 0.990 of the table's ds a path can leave the table's range, so that those experiments replay
with the exact blend and linear derivative tables, the others with the fixed-point table and ratio ones. Needs a B200.

Each gradient must be the one the experiment gets alone (same chains, table and replay; 1e-5 of the largest
entry, as for pixels against single experiments) and the FP64 form's central differences on that table,
to 1e-3 (their own error at h = 1e-3 relative, as elsewhere; the set's float entries add 129 2^-25 / ln 10 per path,
1e-4 of the differences)."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu

F32 = np.float32
SCATTER, SIGMA, H = 10.0, 0.1, 1e-3
MIN_DS, MAX_DS, NDS = 0.1, 0.3, 21                                      # a table at 0.12
EXPERIMENTS = [(64, 0.1225), (64, 0.1175), (40, 0.1215), (130, 0.118)]  # (N, ds): 0.12 is the closest to each
RUN = dict(mu=1.0, num_steps_int=2000, num_curvature_steps=1024, lut_mode=T.LUT_MULTI_DS, num_chains=256, paths_to_skip=30,
           max_sub_chain=32, max_angle=0.05, perturb_seed=8)
PATHS = 256 * 21


def _eps(sigma):
    return float(F32(sigma) * F32(sigma))


def _bc(N, ds):
    S = N * ds
    return T.make_bc((0, 0, 0), (1, 0, 0), (0.55 * S, 0.1 * S, 0), (1, 0, 0), S)


def _params(scatter=SCATTER, sigma=SIGMA, **kw):
    return T.default_params(scatter=float(scatter), eps=_eps(sigma), **{**RUN, **kw})


@pytest.mark.parametrize("order", [(0, 1, 2, 3), (3, 2, 1, 0), (1, 0), (0, 1)])
def test_experiments_on_one_table_take_their_own_replay(order):
    exps = [T.make_experiment(_bc(*EXPERIMENTS[k]), EXPERIMENTS[k][0], SCATTER, _eps(SIGMA), PATHS) for k in order]
    with T.Context(_params(num_segments=16, paths_to_generate=0)) as ctx:
        ctx.multi_ds_tables(MIN_DS, MAX_DS, NDS)
        res, grad, total, _ = ctx.adjoint_batch(exps)
        for i, x in enumerate(exps):
            assert res[i].table_form == T.TABLE_FIXED_NARROW and res[i].steep_bins == 0
            ctx.update(experiment_id=i, bootstrap_seed=i)
            (alone,), g, _, _ = ctx.adjoint_batch([x])
            assert alone.log10_weight == res[i].log10_weight
            assert np.all(np.abs(grad[i] - g[0]) < 1e-5 * np.abs(g[0]).max()), (order, i, grad[i], g[0])
    L = np.array([r.log10_weight for r in res])
    w = 10.0 ** (L - L.max())
    assert total[1] == pytest.approx((w * grad[:, 0]).sum() / w.sum(), rel=1e-12)
    assert total[2] == pytest.approx((w * grad[:, 1]).sum() / w.sum(), rel=1e-12)


@pytest.mark.parametrize("N,ds", EXPERIMENTS)
def test_gradients_match_fp64_differences_on_the_table(N, ds):
    bc = _bc(N, ds)
    other = (64, 0.1175 if ds > 0.12 else 0.1225)   # the other replay on the same table
    exps = [T.make_experiment(_bc(*other), other[0], SCATTER, _eps(SIGMA), PATHS),
            T.make_experiment(bc, N, SCATTER, _eps(SIGMA), PATHS)]
    with T.Context(_params(num_segments=16, paths_to_generate=0)) as ctx:
        ctx.multi_ds_tables(MIN_DS, MAX_DS, NDS)
        res, grad, _, _ = ctx.adjoint_batch(exps)

    def log10w(scatter, sigma):
        p = _params(scatter, sigma, num_segments=N, form=T.FORM_FP64, paths_to_generate=PATHS, num_chains=res[1].num_chains,
                    experiment_id=1, bootstrap_seed=1)
        with T.Context(p) as c:
            c.multi_ds_tables(MIN_DS, MAX_DS, NDS)
            return c.run(bc).log10_weight, float(np.sqrt(np.float64(p.eps))), float(p.scatter)

    hi, lo = log10w(SCATTER * (1 + H), SIGMA), log10w(SCATTER * (1 - H), SIGMA)
    d_mu = (hi[0] - lo[0]) / (hi[2] - lo[2])
    hi, lo = log10w(SCATTER, SIGMA * (1 + H)), log10w(SCATTER, SIGMA * (1 - H))
    d_sigma = (hi[0] - lo[0]) / (hi[1] - lo[1])
    assert abs(grad[1][0] - d_mu) < 1e-3 * abs(d_mu), (grad[1], d_mu)
    assert abs(grad[1][1] - d_sigma) < 1e-3 * abs(d_sigma), (grad[1], d_sigma)
    assert np.all(np.isfinite(grad))
