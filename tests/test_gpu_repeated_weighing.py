"""twisty_weight_paths on one context, call after call: the first large upload goes through the driver, later
ones through the context's pinned ring; sizes around a chunk (1 MB) and the ring's threshold (4 MB), odd
tails, growing and shrinking arrays, each with other paths. Needs a B200.

Every call weighs the same paths as a fresh context does, bit for bit."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu

N, S = 30, 6.0


def _paths(n, seed):
    r = np.random.default_rng(seed)
    t = np.array([0.0, 0.0, 1.0]) + 0.1 * np.cumsum(r.normal(size=(n, N, 3)), axis=1)
    t /= np.linalg.norm(t, axis=2, keepdims=True)
    pos = np.zeros((n, N + 1, 3), np.float32)
    pos[:, 1:] = np.cumsum(t * (S / N), axis=1)
    return pos


@pytest.mark.parametrize("form", [T.FORM_COMPENSATED, T.FORM_PLAIN_FP32])
def test_repeated_weighing_matches_fresh_contexts(form):
    p = T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=1024, form=form)
    bc = T.make_bc((0, 0, 0), (0, 0, 1), (0, 0, 4), (0, 0, 1), S)
    row = 12 * (N + 1)
    mb = 1 << 20
    sizes = [5 * mb // row, 3, 4 * mb // row, 4 * mb // row + 1, 4 * mb // row - 1, 9 * mb // row + 7, 33 * mb // row, 1]
    with T.Context(p) as ctx:
        for i, n in enumerate(sizes):
            pos = _paths(n, i)
            w, v, b = ctx.weight_paths(bc, pos, form, want_bins=(i % 2 == 0))
            with T.Context(p) as fresh:
                w2, v2, b2 = fresh.weight_paths(bc, pos, form, want_bins=(i % 2 == 0))
            assert np.array_equal(w, w2) and np.array_equal(v, v2) and np.all(v == 1)
            assert b is None or np.array_equal(b, b2)
