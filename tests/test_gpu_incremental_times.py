"""Device times of incremental passes relative to the full recompute of the same chains on 32 lanes: their single-tangent
reads want the unpaired layout. Needs a B200.

Measured at N = 530, 768, 1024 (2^29 path-segments, 2048 bins, a recompute every 64 weighted steps): 0.685, 0.587 and 0.533
of the full recompute's time; with the paired layout 0.790, 0.666 and 0.597. The lines lie between."""
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


def _min_ms(N, resync):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.6 * S, 0.1, 0), (1, 0, 0), S)
    with T.Context(T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=2048,
                                    perturb_seed=3, paths_to_generate=(1 << 29) // N, paths_to_skip=30, max_sub_chain=32,
                                    max_angle=0.05, incremental_resync=resync)) as ctx:
        ctx.run(bc)
        return min(ctx.run(bc).perturb_ms for _ in range(5))


@pytest.mark.parametrize("N,line", [(530, 0.735), (768, 0.625), (1024, 0.565)])
def test_incremental_passes_keep_their_pace(N, line):
    incremental, full = _min_ms(N, 64), _min_ms(N, 0)
    assert incremental < line * full, (incremental, full)
