"""The M-segment kernel's paths one by one: a run of P paths against P runs of one path each
(chain_offset numbers the paths), for spans that close in twos and in threes and path counts
around a block's and a slice's. Needs a B200.

The same path gives the same weight whichever thread and launch builds it, so the mean differs only by
the order of FP64 sums: 1e-12 in log10."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


def _params(N, form, paths, offset=0):
    return T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=1024,
                            paths_to_generate=paths, perturb_seed=5, form=form, chain_offset=offset, absorption=0.05)


@pytest.mark.parametrize("form", [T.FORM_COMPENSATED, T.FORM_PLAIN_FP32])
@pytest.mark.parametrize("N,paths", [(6, 1), (8, 129), (10, 128), (26, 200), (66, 131), (98, 64)])
def test_a_run_is_the_mean_of_its_paths(N, paths, form):
    bc = T.make_bc((0, 0, 0), (0, 0, 1), (0, 0, 0.6 * 0.3 * N), (0, 0, 1), 0.3 * N)
    with T.Context(_params(N, form, paths)) as ctx:
        whole = ctx.run_msegment(bc)
        logs = []
        for i in range(paths):
            ctx.set_params(_params(N, form, 1, i))
            r = ctx.run_msegment(bc)
            if r.total_paths:
                logs.append(r.log10_mean_weight)
    logs = np.array(logs)
    assert whole.total_paths == logs.size and whole.failed_paths == paths - logs.size
    want = logs.max() + np.log10(np.mean(10.0 ** (logs - logs.max())))
    assert abs(whole.log10_mean_weight - want) < 1e-12 * max(1.0, abs(want))


@pytest.mark.parametrize("paths", [16383, 16385, 120000])
def test_runs_of_two_halves_combine(paths):
    """Paths 0..P-1 and P..2P-1 as runs of their own, against one run of 2P (several paths per thread)."""
    N = 34
    bc = T.make_bc((0, 0, 0), (0, 0, 1), (0, 0, 7), (0, 0, 1), 12.0)
    with T.Context(_params(N, T.FORM_COMPENSATED, 2 * paths)) as ctx:
        whole = ctx.run_msegment(bc)
        half = []
        for k in range(2):
            ctx.set_params(_params(N, T.FORM_COMPENSATED, paths, k))
            half.append(ctx.run_msegment(bc))
    assert whole.total_paths == half[0].total_paths + half[1].total_paths
    m = max(h.log10_mean_weight for h in half)
    want = m + np.log10(sum(h.total_paths * 10.0 ** (h.log10_mean_weight - m) for h in half) / whole.total_paths)
    assert abs(whole.log10_mean_weight - want) < 1e-11
