"""M-segment paths whose spans close in threes (N - 2 = 6, 12, 24, ...) and in twos, which kernels of their own build.
Needs a B200.

Both forms build the same paths from the same draws, so the same paths fail, and the mean weights agree to the
forms' own difference: the plain form's float blend (2.6e-8 a segment) and the compensated one's secant and
fixed point (under 1.1e-7)."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


def _run(N, form, paths, f=0.6, repeat=1):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (0, 0, 1), (0, 0, f * S), (0, 0, 1), S)
    with T.Context(T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=2048,
                                    paths_to_generate=paths, perturb_seed=5, form=form)) as ctx:
        rs = [ctx.run_msegment(bc) for _ in range(repeat)]
    return rs[0], min(r.perturb_ms for r in rs)


@pytest.mark.parametrize("f", [0.3, 0.9])
@pytest.mark.parametrize("N", [6, 8, 14, 18, 26, 50, 98, 130, 194, 386, 514, 770])
def test_both_forms_weigh_the_same_paths(N, f):
    paths = 100_000 if N < 100 else 20_000
    plain, _ = _run(N, T.FORM_PLAIN_FP32, paths, f)
    comp, _ = _run(N, T.FORM_COMPENSATED, paths, f)
    assert plain.total_paths + plain.failed_paths == paths
    assert comp.total_paths == plain.total_paths and comp.failed_paths == plain.failed_paths
    # a bin edge between two roundings of a curvature moves one segment's weight by a bin: a path in 1000 at most
    # is far off by that, 1e-3 of it, so the mean by 1e-6
    assert abs(comp.log10_mean_weight - plain.log10_mean_weight) < N * 1.4e-7 + 1e-6


@pytest.mark.parametrize("N", [194, 386])
def test_compensated_paths_of_threes_keep_their_pace(N):
    """Device times at 2^26 path-segments, compensated over plain: 0.83 to 0.85; 1.25 to 1.3 with the leaves of both
    kinds in one kernel."""
    paths = (1 << 26) // N
    _, plain = _run(N, T.FORM_PLAIN_FP32, paths, repeat=4)
    _, comp = _run(N, T.FORM_COMPENSATED, paths, repeat=4)
    assert comp < 1.05 * plain, (comp, plain)
