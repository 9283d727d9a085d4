"""Time of a weights-only replay (the path-weight histogram) relative to the fixed-point pass of the same chains: it runs the
pass's recompute and one weight per path to memory. Needs a B200.

Measured at N = 384, 700, 896 (2^29 path-segments, 2048 bins): the call takes 1.50, 1.66, 1.66 times the pass's device
time; with the loads of a lane's segments hoisted until they spilled 2.10, 2.84, 2.39. The line lies between."""
import time

import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [384, 700, 896])
def test_replays_keep_their_pace(N):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.6 * S, 0.1, 0), (1, 0, 0), S)
    with T.Context(T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=2048,
                                    perturb_seed=3, paths_to_generate=(1 << 29) // N, paths_to_skip=30, max_sub_chain=32,
                                    max_angle=0.05)) as ctx:
        ctx.run(bc)
        fixed = min(ctx.run(bc).perturb_ms for _ in range(5))
        ctx.weight_histogram(bc)
        ms = []
        for _ in range(5):
            t0 = time.perf_counter()
            counts = ctx.weight_histogram(bc)
            ms.append(1e3 * (time.perf_counter() - t0))
    assert int(counts.sum()) == (1 << 29) // N
    assert min(ms) < 1.9 * fixed, (min(ms), fixed)
