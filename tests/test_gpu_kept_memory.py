"""Device memory a context keeps between calls: the calls' buffers 256 MB together, the M-segment estimator's 512 MB
(its columns take up to 384 of them); all of it is given back with the context. Needs a B200."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu

MB = 1 << 20
SLACK = 16 * MB      # tables, allocation granularity


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_kept_memory_is_bounded_and_given_back():
    N, P = 8, 2_300_000
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.6 * S, 0.1, 0), (1, 0, 0), S)
    p = dict(mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=512, max_sub_chain=32, max_angle=0.05)
    walk = np.random.default_rng(3).normal(size=(P, N + 1, 3)).astype(np.float32)
    with T.Context(T.default_params(num_segments=10, paths_to_generate=1000, **p)) as warm:   # modules, lazy allocations
        warm.run_msegment(T.make_bc((0, 0, 0), (1, 0, 0), (0.7, 0.1, 0), (1, 0, 0), 1.2))
        warm.weight_paths(T.make_bc((0, 0, 0), (1, 0, 0), (0.7, 0.1, 0), (1, 0, 0), 1.2), np.zeros((1, 11, 3), np.float32), want_bins=True)
    before = _free()
    with T.Context(T.default_params(num_segments=N, paths_to_generate=1000, **p)) as ctx:
        ctx.weight_paths(bc, walk[:100], want_bins=True)
        for _ in range(2):
            w, v, b = ctx.weight_paths(bc, walk, want_bins=True)   # 248 MB of points, 64 of bins, 20 of weights
            assert before - _free() <= 256 * MB + SLACK
        w2, v2, b2 = ctx.weight_paths(bc, walk[1000:2000], want_bins=True)
        assert np.array_equal(w[1000:2000], w2) and np.array_equal(v[1000:2000], v2) and np.array_equal(b[1000:2000], b2)
    assert before - _free() <= SLACK
    S = 0.12 * 258
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.6 * S, 0.1, 0), (1, 0, 0), S)
    with T.Context(T.default_params(num_segments=258, paths_to_generate=1 << 18, **p)) as ctx:
        ctx.run_msegment(bc)
        assert before - _free() <= 512 * MB + SLACK
    assert before - _free() <= SLACK
