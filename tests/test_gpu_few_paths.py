"""Passes of fewer paths than the default grid has chains: the chains are spread over the SMs on smaller CTAs, and stay
the ones that the same pass makes when the chain count is asked for. Needs a B200.

One path per chain either way; the CTA's warp count enters no arithmetic, so the results are the same bits."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [4, 16, 66, 258, 1024])
@pytest.mark.parametrize("paths", [1, 149, 2369, 4737])
def test_default_spread_keeps_the_chains(N, paths):
    S = max(0.12 * N, 1.0)
    kw = dict(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=1024,
              paths_to_generate=paths, paths_to_skip=7, max_sub_chain=32, max_angle=0.1, perturb_seed=21)
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.55 * S, 0.1 * S, 0), (1, 0, 0), S)
    out = []
    for chains in (0, paths):
        with T.Context(T.default_params(num_chains=chains, **kw)) as ctx:
            r = ctx.run(bc)
            assert r.total_paths + r.failed_paths == paths
            out.append((r.num_chains, r.log10_weight, ctx.chain_results(r.num_chains)))
    if out[0][0] == out[1][0]:
        assert out[0][1] == out[1][1] and np.array_equal(out[0][2][0], out[1][2][0]) and np.array_equal(out[0][2][1], out[1][2][1])
    else:   # the grid has fewer chains than there are paths: the default gives each several
        assert out[0][0] < paths and paths > 148 * 4
