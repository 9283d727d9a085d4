"""Incremental passes through steep bins, on shapes of every layout: paths that the fixed-point table cannot weigh are weighed
again from the chain's own state. Needs a B200.

The same moves weighed by full recomputes and incrementally: no path is lost either way, and the incremental total is off
by its rounded terms, two of half a unit 2^-22 at most per step over up to 7 steps: 1e-6 in log10 with the
running sums' rounding."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resync", [2, 8])
@pytest.mark.parametrize("G,SPL,N", [(1, 16, 13), (4, 9, 36), (4, 16, 60), (8, 16, 125), (16, 16, 256), (32, 4, 98), (32, 4, 128), (32, 17, 514),
                                     (32, 20, 640), (32, 28, 800), (32, 32, 1024)])
def test_incremental_steep_paths(G, SPL, N, resync):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (0, 0, 1), (0, 0.1, 0.6 * S), (0, 0, 1), S)
    kw = dict(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=1024, form=T.FORM_COMPENSATED,
              num_chains=48, paths_to_generate=48 * 40, paths_to_skip=20, max_sub_chain=32, max_angle=0.1, perturb_seed=5,
              comp_group=G, comp_spl=SPL, comp_warps=4)
    with T.Context(T.default_params(**kw)) as ctx:
        lut, info = ctx.build_lut(float(np.float32(S) / np.float32(N)))
        pos, _, _ = ctx.export_paths(bc, None, 400)
        _, _, bins = ctx.weight_paths(bc, pos, want_bins=True)
        c = max(int(np.median(bins)), 2)
        steep = lut.copy()
        steep[c:c + 6:2] *= 1.5
        steep[c + 1:c + 6:2] *= 0.5
        ctx.set_lut(steep, info)
        full = ctx.run(bc)
        ctx.update(incremental_resync=resync)
        incr = [ctx.run(bc) for _ in range(2)]
    assert full.steep_bins >= 5 and full.kernel_shape == (G << 8 | SPL)
    for r in incr:
        assert r.total_paths == full.total_paths == 48 * 40 and r.failed_paths == full.failed_paths == 0
        assert abs(r.log10_weight - full.log10_weight) < 1e-6, (r.log10_weight, full.log10_weight)
