"""Paths through steep bins are weighed with the exact blend's own arithmetic: the segments of a lane in order, whatever
the shape's layout. Needs a B200.

The same chains (the moves do not see the weights) are exported twice: with a table of a few steep bins, which keeps its
fixed-point form, and with the same table plus a zigzag over entries that no path blends, which takes the exact
blend for every path. A path through a steep bin is the same sum both times, once rounded to the fixed point:
within half a unit 2^-s, and 1e-12 for the doubles."""
import math

import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu

BINS = 1024


@pytest.mark.parametrize("G,SPL,N", [(1, 16, 13), (1, 24, 24), (4, 5, 18), (4, 12, 45), (4, 16, 64), (4, 17, 66), (8, 16, 125),
                                     (16, 16, 256), (32, 4, 100), (32, 8, 256), (32, 17, 514), (32, 32, 701)])
def test_steep_paths_equal_the_exact_blend(G, SPL, N):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (0, 0, 1), (0, 0.1, 0.6 * S), (0, 0, 1), S)
    p = T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=BINS,
                         form=T.FORM_COMPENSATED, num_chains=48, paths_to_generate=48 * 8, paths_to_skip=20, max_sub_chain=32,
                         max_angle=0.1, perturb_seed=5, comp_group=G, comp_spl=SPL, comp_warps=4)
    with T.Context(p) as ctx:
        lut, info = ctx.build_lut(float(np.float32(S) / np.float32(N)))
        pos, _, r = ctx.export_paths(bc, None, 48 * 8)
        assert r.kernel_shape == (G << 8 | SPL)
        _, _, bins = ctx.weight_paths(bc, pos, want_bins=True)
        c = max(int(np.median(bins)), 2)
        met = np.zeros(BINS + 4, bool)        # bins that a path is in or within two of
        for d in range(-2, 3):
            met[np.clip(bins + d, 0, BINS + 3)] = True
        steep = lut.copy()
        steep[c:c + 6:2] *= 1.5
        steep[c + 1:c + 6:2] *= 0.5
        ctx.set_lut(steep, info)
        pos_s, w_s, r_s = ctx.export_paths(bc, None, 48 * 8)
        exact = steep.copy()
        free = [i for i in range(c + 20, BINS) if not met[i] and not met[i - 1]]
        exact[free[::2]] *= 4.0
        ctx.set_lut(exact, info)
        pos_e, w_e, r_e = ctx.export_paths(bc, None, 48 * 8)
    assert r_s.table_form in (T.TABLE_FIXED_NARROW, T.TABLE_FIXED_WIDE) and r_s.steep_bins >= 5
    assert r_e.table_form == T.TABLE_EXACT_BLEND
    assert np.array_equal(pos_s, pos_e) and np.array_equal(pos_s, pos)
    # bins c - 1 .. c + 5 are steep: a path in c .. c + 4 meets one even if an end of its bin rounds the other way
    hit = np.any((bins >= c) & (bins <= c + 4), axis=1)
    assert hit.sum() >= 20
    lg = np.log10(steep.astype(np.float64))
    span, s = lg.max() - lg.min(), 30
    # N + 1 entries below 2^31 (narrow totals), or 32 below 2^32 (wide ones)
    cap = (2.0 ** 31 - 1) / (N + 1) if r_s.table_form == T.TABLE_FIXED_NARROW else (2.0 ** 32 - 1) / 32
    while span * 2.0 ** s + 65.0 > math.floor(cap):
        s -= 1
    assert s >= 22
    assert np.abs(w_s - w_e)[hit].max() <= 0.5 * 2.0 ** -s + 1e-12
