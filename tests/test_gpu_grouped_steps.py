"""Chains whose weighted steps do not fill the groups of four that the forward passes sum together,
against the FP64 form on the same proposals, through the C ABI. Needs a B200.

Groups of 4 lanes and more add four steps' path totals at a time and finish with a partial group; the last
chain of a pass stops earlier than the others of its warp. A step lost, counted twice or summed
into another would move a chain's sum by about log10 of the steps (0.1 and more). The tolerance is
the one of the shape sweep: 1.5e-7 |log10 w| for the FP32 trajectory plus 1e-5."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


# 4 x 4 and 4 x 17 (N = 16, 66), 8 x 17, 16 x 17, 32 x 24 with 64-bit totals (N = 130, 258, 700)
@pytest.mark.parametrize("N", [16, 66, 130, 258, 700])
@pytest.mark.parametrize("steps,short", [(1, 0), (2, 1), (3, 2), (4, 1), (5, 0), (6, 3), (9, 7)])
def test_partial_groups_of_steps_match_fp64(N, steps, short):
    chains = 300
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.55 * S, 0.1 * S, 0), (1, 0, 0), S)
    out = {}
    for form in (T.FORM_COMPENSATED, T.FORM_FP64):
        p = T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000,
                             num_curvature_steps=2048, form=form, lut_mode=T.LUT_FP64, perturb_seed=11, num_chains=chains,
                             paths_to_generate=chains * steps - short, paths_to_skip=7, max_sub_chain=32, max_angle=0.05)
        with T.Context(p) as ctx:
            r = ctx.run(bc)
            lw, valid = ctx.chain_results(r.num_chains)
        assert r.num_chains == chains and r.failed_paths == 0 and r.total_paths == chains * steps - short
        assert valid[0] == steps and valid[-1] == steps - short
        out[form] = lw
    a, b = out[T.FORM_COMPENSATED], out[T.FORM_FP64]
    assert np.all(np.abs(a - b) < 1.5e-7 * np.abs(b) + 1e-5)
