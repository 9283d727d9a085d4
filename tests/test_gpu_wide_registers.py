"""The 28- and 32-segment shapes on 32 lanes at both sides of 16 warps per CTA, where the forward pass moves to a build
with fewer registers, full and padded chains, the table staged and through L1, with and without steep bins. Needs a
B200.

Both builds compile the same arithmetic: each chain's sum has the same bits."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [0.01, 0.0025])
@pytest.mark.parametrize("N,spl,few,many,memory", [(769, 28, 16, 17, 0), (896, 28, 16, 20, 2), (850, 28, 7, 18, 0), (897, 32, 12, 17, 2),
                                                   (1000, 32, 16, 17, 2), (1024, 32, 12, 17, 2)])
def test_both_builds_give_the_same_chains(N, spl, few, many, memory, eps):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.55 * S, 0.1 * S, 0), (1, 0, 0), S)
    out = []
    for warps in (few, many):
        p = T.default_params(num_segments=N, mu=1.0, eps=eps, scatter=10.0, num_steps_int=2000, num_curvature_steps=512,
                             paths_to_generate=100 * 40, num_chains=100, paths_to_skip=9, max_sub_chain=32, max_angle=0.3, perturb_seed=6,
                             comp_group=32, comp_spl=spl, comp_warps=warps, comp_table_memory=memory)
        with T.Context(p) as ctx:
            r = ctx.run(bc)
            assert r.total_paths + r.failed_paths == 4000
            out.append(ctx.chain_results(r.num_chains))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
