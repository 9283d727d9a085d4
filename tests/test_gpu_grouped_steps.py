"""Chains whose weighted steps do not fill the groups of four that the forward passes sum together,
against the same chains' path weights as the export replay gives them one by one, through the
C ABI. Needs a B200.

Groups of 4 lanes and more add four steps' path totals at a time and finish with a partial group; the last
chain of a pass stops earlier than the others of its warp. The export replays the same chains with a total
per step, so a chain's sum differs from the log-sum-exp of its exported weights only by the
rounding of the running sum: a float exponential of 2^-22 relative error per path and a compensated
float sum, under 1e-6 in log10 together. A step lost, counted twice or summed into another
would move it by 0.04 and more."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


# 4 x 4 and 4 x 17 (N = 16, 66), 8 x 17, 16 x 17, 32 x 24 with 64-bit totals (N = 130, 258, 700)
@pytest.mark.parametrize("N", [16, 66, 130, 258, 700])
@pytest.mark.parametrize("steps,short", [(1, 0), (2, 1), (3, 2), (4, 1), (5, 0), (6, 3), (9, 7)])
def test_partial_groups_of_steps_match_the_paths(N, steps, short):
    chains = 300
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.55 * S, 0.1 * S, 0), (1, 0, 0), S)
    paths = chains * steps - short
    p = T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=2048,
                         form=T.FORM_COMPENSATED, lut_mode=T.LUT_FP64, perturb_seed=11, num_chains=chains,
                         paths_to_generate=paths, paths_to_skip=7, max_sub_chain=32, max_angle=0.05)
    with T.Context(p) as ctx:
        r = ctx.run(bc)
        sums, valid = ctx.chain_results(r.num_chains)
        _, w, _ = ctx.export_paths(bc, None, paths)
    assert r.num_chains == chains and r.failed_paths == 0 and r.total_paths == paths == w.size
    assert np.all(valid[:-1] == steps) and valid[-1] == steps - short
    for i in range(chains):
        x = w[i * steps:(i + 1) * steps]
        want = x.max() + np.log10(np.sum(10.0 ** (x - x.max())))
        assert abs(sums[i] - r.log10_normalizer - want) < 1e-6, i
