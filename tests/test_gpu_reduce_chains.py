"""The log-sum-exp reduction of a pass's chains at both sides of the chain count where it moves from one CTA to
a cluster of 8 (4096), around whole rounds of the cluster (8 x 1024 chains), against NumPy's reduction of the same
chain sums. Needs a B200.

Both sides add n positive doubles that are each right to a few ulp of exp10 (rel. 1e-15): the sums agree to
d = 1e-15 + n 2^-53 at the very worst, log10 of the sum to d / ln 10 and the roundings of doubles of magnitude 64
(four, each 7e-15). The relative standard error comes from the sum of squares minus n mean^2, so with the chains'
relative variance v its square is off by 2 d (1 + 1 / v) at most; twice that here."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chains", [1, 2, 31, 1023, 4095, 4096, 4097, 8191, 8192, 8193, 20000])
def test_reduction_matches_numpy(chains):
    p = T.default_params(num_segments=30, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=1024,
                         num_chains=chains, paths_to_generate=chains * 8, paths_to_skip=16, max_sub_chain=16, perturb_seed=9)
    with T.Context(p) as ctx:
        r = ctx.run(T.make_bc((0, 0, 0), (1, 0, 0), (2.6, 0.3, 0), (1, 0, 0), 3.6))
        lw, valid = ctx.chain_results(r.num_chains)
    assert r.num_chains == chains and r.total_paths == chains * 8
    assert int(valid.sum()) == r.total_paths - r.failed_paths
    x = 10.0 ** (lw - lw.max())
    d = 1e-15 + chains * 2.0 ** -53
    assert abs(r.log10_weight - (lw.max() + np.log10(x.sum()))) < d + 2.8e-14
    if chains > 1:
        v = x.var(ddof=1) / x.mean() ** 2
        assert abs(r.rel_std_error ** 2 * chains - v) <= 4 * d * (1 + v)
    else:
        assert np.isnan(r.rel_std_error)
