"""Device times of the exact-blend and receiver-shifted passes relative to the fixed-point pass of the same chains:
they walk their segments in order, whatever layout the fixed-point form prefers. Needs a B200.

Measured at N = 768, 896, 1024 (2^28 path-segments, 2048 bins), times the fixed-point pass: exact 1.33, 1.40, 1.39 and
shifted 1.69, 1.78, 1.82; with the ordered walk over paired tangents 1.62, 1.76, 1.85 and 2.38, 2.51, 2.82. The lines lie
between the two."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


def _min_ms(ctx, bc):
    ctx.run(bc)
    return min(ctx.run(bc).perturb_ms for _ in range(5))


@pytest.mark.parametrize("N", [768, 896, 1024])
def test_ordered_walks_keep_their_pace(N):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.6 * S, 0.1, 0), (1, 0, 0), S)
    p = dict(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=2048, perturb_seed=3,
             paths_to_generate=(1 << 28) // N, paths_to_skip=30, max_sub_chain=32, max_angle=0.05)
    with T.Context(T.default_params(**p)) as ctx:
        fixed = _min_ms(ctx, bc)
        lut, info = ctx.build_lut(float(np.float32(S) / np.float32(N)))
        lut[-1] = 0.0
        ctx.set_lut(lut, info)
        exact = _min_ms(ctx, bc)
    with T.Context(T.default_params(eval_end_shift=(0.01, 0.0, 0.0), **p)) as ctx:
        shifted = _min_ms(ctx, bc)
    assert exact < 1.5 * fixed and shifted < 2.1 * fixed, (fixed, exact, shifted)
