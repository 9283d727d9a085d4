"""The single run's tables (one cluster launch: finalisation, fixed-point and linear forms) against the
batched run's (a CTA per table) at table sizes around the cluster's 8192 threads, and on caller's
tables that are steep, have non-positive entries or are as small as two bins. Needs a B200.

Both follow the same rules on the same float table, so the form and the steep bins agree exactly; the
weights to 1e-6 in log10, the batched runs' own tolerance against single runs."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


def _params(bins, eps, **kw):
    base = dict(num_segments=66, mu=1.0, eps=eps, scatter=10.0, num_steps_int=2000, num_curvature_steps=bins,
                form=T.FORM_COMPENSATED, lut_mode=T.LUT_FP64, perturb_seed=7, bootstrap_seed=3, num_chains=256, paths_to_generate=256 * 40,
                paths_to_skip=10, max_sub_chain=32, max_angle=0.05)
    base.update(kw)
    return T.default_params(**base)


BC = ((0, 0, 0), (1, 0, 0), (8, 0, 0), (1, 0, 0), 10.0)


@pytest.mark.parametrize("eps", [0.01, 0.05 ** 2])
@pytest.mark.parametrize("bins", [64, 1023, 8191, 8192, 8193, 16385, 20000])
def test_single_tables_match_batched(bins, eps):
    bc = T.make_bc(*BC)
    with T.Context(_params(bins, eps)) as ctx:
        one = ctx.run(bc)
        many, = ctx.run_batch([T.make_experiment(bc, 66, 10.0, eps, 256 * 40)])
    assert one.total_paths == many.total_paths and one.num_chains == many.num_chains
    assert one.steep_bins == many.steep_bins and one.table_form == many.table_form
    assert abs(one.log10_weight - many.log10_weight) < 1e-6


@pytest.mark.parametrize("bins", [2, 3, 257, 8200])
def test_caller_tables_take_the_right_form(bins):
    bc = T.make_bc(*BC)
    with T.Context(_params(bins, 0.01)) as ctx:
        lut, info = ctx.build_lut(10.0 / 66)
        assert np.all(lut > 0) and info.min_segment_weight == lut.min() and info.max_segment_weight == lut.max()
        r = ctx.run(bc)
        bad = lut.copy()
        bad[bins // 2] = 0.0
        ctx.set_lut(bad, info)
        z = ctx.run(bc)
        ctx.set_lut(lut, info)   # the same table again, given by the caller
        again = ctx.run(bc)
    assert z.table_form == T.TABLE_EXACT_BLEND and z.steep_bins <= bins
    assert again.table_form == r.table_form and again.steep_bins == r.steep_bins
    assert again.log10_weight == r.log10_weight
