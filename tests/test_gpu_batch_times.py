"""Device times of batches of padded chains relative to batches that fill their shape's slots: the same slots, and one
weight more or less per lane. Needs a B200.

Measured for 24 experiments of 2^14 paths (2048 bins): N = 180 takes 1.09 times as long per path as 192, 350 1.09 times 384,
400 1.04 times 448; with sums of four paths in flight, for which the batched kernels have no registers, 1.32, 1.36, 1.45.
The line lies between."""
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


def _min_ms(N):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.6 * S, 0.1, 0), (1, 0, 0), S)
    p = T.default_params(num_segments=16, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=2048, perturb_seed=3,
                         bootstrap_seed=4, paths_to_generate=0, paths_to_skip=30, max_sub_chain=32, max_angle=0.05)
    with T.Context(p) as ctx:
        exps = [T.make_experiment(bc, N, 10.0, 0.01, 1 << 14) for _ in range(24)]
        ctx.run_batch(exps)
        return min(ctx.run_batch(exps)[0].perturb_ms for _ in range(5))


@pytest.mark.parametrize("padded,full", [(180, 192), (350, 384), (400, 448)])
def test_padded_batches_keep_their_pace(padded, full):
    a, b = _min_ms(padded), _min_ms(full)
    assert a < 1.2 * b, (a, b)
