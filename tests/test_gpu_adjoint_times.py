"""Time of the adjoint replay relative to the forward pass of the same chains, for shapes of 32 warps: the replay runs the
pass's CTAs as they are, not on fewer warps and a nearly empty second wave. Needs a B200.

Measured at 2^30 path-segments (2048 bins), the call over the pass's device time: 1.74, 1.85 and 1.59 at N = 28, 36 and 72
with the fixed-point replay, 1.93, 1.85 and 1.85 with the exact one; on 24 warps 2.55, 2.74, 2.39 and 2.98, 2.83, 2.83. The
line lies between."""
import time

import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps,scatter", [(0.01, 10.0), (0.0025, 40.0)])     # fixed-point and exact replays
@pytest.mark.parametrize("N", [28, 36, 72])
def test_replays_of_wide_ctas_keep_their_pace(N, eps, scatter):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.6 * S, 0.1, 0), (1, 0, 0), S)
    with T.Context(T.default_params(num_segments=N, mu=1.0, eps=eps, scatter=scatter, num_steps_int=2000, num_curvature_steps=2048,
                                    perturb_seed=3, bootstrap_seed=4, paths_to_generate=(1 << 30) // N, paths_to_skip=30,
                                    max_sub_chain=32, max_angle=0.05)) as ctx:
        fwd = ctx.run(bc)
        forward = min(ctx.run(bc).perturb_ms for _ in range(4))
        ctx.adjoint(bc, fwd)
        ms = []
        for _ in range(4):
            t0 = time.perf_counter()
            ctx.adjoint(bc, fwd)
            ms.append(1e3 * (time.perf_counter() - t0))
    assert (fwd.steep_bins > 0) == (eps < 0.01)
    assert min(ms) < 2.1 * forward, (min(ms), forward)
