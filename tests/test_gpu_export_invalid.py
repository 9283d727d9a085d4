"""Export with invalid paths scattered among the valid ones: a table entry below zero makes every path that blends it
invalid, and the export gives the others, in order, as the same chains' export through the table without it gives
them, in a time that does not grow with the number of gaps. Needs a B200."""
import time

import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu

N, CHAINS, STEPS = 8, 64, 160      # each move changes two of seven curvatures: validity changes often


def _min_s(f, n=5):
    ts = []
    for _ in range(n):
        t0 = time.perf_counter()
        f()
        ts.append(time.perf_counter() - t0)
    return min(ts)


@pytest.mark.parametrize("form", [T.FORM_COMPENSATED, T.FORM_PLAIN_FP32])
def test_export_skips_scattered_invalid_paths(form, tmp_path):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (0, 0, 1), (0, 0.1, 0.6 * S), (0, 0, 1), S)
    p = T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=1024, form=form,
                         num_chains=CHAINS, paths_to_generate=CHAINS * STEPS, paths_to_skip=5, max_sub_chain=32, max_angle=3.14,
                         perturb_seed=5)
    with T.Context(p) as ctx:
        lut, info = ctx.build_lut(float(np.float32(S) / np.float32(N)))
        clean = lut.copy()
        clean[-1] = 0.0                       # above every curvature met: the exact blend, no path invalid
        ctx.set_lut(clean, info)
        pos, w, r = ctx.export_paths(bc, None, CHAINS * STEPS)
        assert r.failed_paths == 0 and pos.shape[0] == CHAINS * STEPS
        _, _, bins = ctx.weight_paths(bc, pos, want_bins=True)
        lo, hi = np.quantile(bins, [0.45, 0.55]).astype(int)   # a tenth of the curvatures: half of the paths
        holes = clean.copy()
        holes[lo:hi + 1] = -1.0
        ctx.set_lut(holes, info)
        got, gw, gr = ctx.export_paths(bc, None, CHAINS * STEPS)
        some, sw, _ = ctx.export_paths(bc, None, 1234)
        filed, fw, _ = ctx.export_paths(bc, str(tmp_path), 1234)
        slow = _min_s(lambda: ctx.export_paths(bc, None, CHAINS * STEPS))
        ctx.set_lut(clean, info)
        fast = _min_s(lambda: ctx.export_paths(bc, None, CHAINS * STEPS))
    # the valid paths are a subsequence of the chains' paths, and there are as many gaps as the case is about
    n = got.shape[0]
    assert n == gr.total_paths and gr.failed_paths == CHAINS * STEPS - n
    at, idx = -1, []
    for i in range(n):
        at += 1
        while not np.array_equal(pos[at], got[i]):
            at += 1
        idx.append(at)
    idx = np.array(idx)
    assert np.sum(np.diff(idx) > 1) > 300
    # 1234 paths are looked for in the first 8 chains
    m = np.sum(idx < 8 * STEPS)
    assert np.array_equal(some, got[:m]) and np.array_equal(sw, gw[:m])
    assert np.array_equal(filed, got[:m]) and np.array_equal(fw, gw[:m])
    assert slow < 2.0 * fast, (slow, fast)
