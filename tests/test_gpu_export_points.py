"""Exported points, made by a warp per path after the replay: the paths of every lane group and of padded and full
chains, with both table forms. Needs a B200.

The points are x_0 plus prefix sums of l_s t_s in double, rounded once to float: each of a segment's two end points is
within 2^-24 of its magnitude, the tangents are unit and the lengths are the initial path's to 1e-6, so a segment
of an exported path is as long as the initial path's to 1e-6 S / N + 2^-22 max|x|. The last point, which the moves keep,
is off by the drift of N float tangents over 43 moves of 2^-20 at most."""
import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zero", [False, True])       # True: a table with a zero entry takes the exact blend
@pytest.mark.parametrize("N,chains,paths", [(4, 3, 7), (13, 33, 100), (32, 100, 1000), (48, 5, 64), (66, 300, 1500), (128, 9, 90),
                                            (130, 40, 81), (258, 7, 50), (512, 3, 31), (701, 2, 11), (1024, 2, 9)])
def test_exported_points(N, chains, paths, zero):
    S = 0.12 * N
    x0 = np.array([0.5, 0.0, -3.0])
    p = T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=1024,
                         num_chains=chains, paths_to_generate=chains * 40, paths_to_skip=3, max_sub_chain=32, max_angle=0.1, perturb_seed=5)
    bc = T.make_bc(tuple(x0), (0, 0, 1), (0.5, 0, -3 + 0.6 * S), (0, 0, 1), S)
    init = np.diff(T.bootstrap_curve(p, bc).astype(np.float64).reshape(N + 1, 3), axis=0)
    with T.Context(p) as ctx:
        if zero:
            lut, info = ctx.build_lut(S / N)
            lut[-2] = 0
            ctx.set_lut(lut, info)
        pos, w, r = ctx.export_paths(bc, None, paths)
        again, w_again, _ = ctx.export_paths(bc, None, paths)
    assert pos.shape == (min(paths, chains * 40), N + 1, 3) and r.failed_paths == 0
    assert np.array_equal(pos, again) and np.array_equal(w, w_again)
    d = pos.astype(np.float64)
    assert np.all(d[:, 0] == x0)
    mag = np.abs(d).max()
    ln = np.linalg.norm(np.diff(d, axis=1), axis=2)
    assert np.abs(ln - np.linalg.norm(init, axis=1)).max() <= 1e-6 * S / N + 2.0 ** -22 * mag
    end = d[:, -1] - d[0, -1]
    assert np.abs(end).max() <= 43 * N * 2.0 ** -20 * S / N
    assert np.unique(d.reshape(d.shape[0], -1), axis=0).shape[0] > 1


@pytest.mark.parametrize("chains", [5, 700, 0])
def test_replay_beside_the_pass(chains):
    """The replay runs beside the pass: exports that grow, shrink and take every chain, with passes between them on
    one context, give the bits of fresh contexts, and the pass's result is the plain run's."""
    N, S = 66, 7.92
    p = T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=1024,
                         num_chains=chains, paths_to_generate=6000, paths_to_skip=11, max_sub_chain=32, max_angle=0.1, perturb_seed=8)
    bcs = [T.make_bc((0, 0, 0), (0, 0, 1), (0, 0, f * S), (0, 0, 1), S) for f in (0.6, 0.7)]
    with T.Context(p) as ctx:
        for i, n in enumerate((1, 3000, 10, 6000, 6000, 1200)):
            bc = bcs[i % 2]
            pos, w, r = ctx.export_paths(bc, None, n)
            q = ctx.run(bc)
            with T.Context(p) as fresh:
                pos2, w2, r2 = fresh.export_paths(bc, None, n)
            assert w.size == n and np.array_equal(pos, pos2) and np.array_equal(w, w2)
            assert r.log10_weight == r2.log10_weight == q.log10_weight and r.total_paths == q.total_paths == 6000
            assert r.rel_std_error == q.rel_std_error and r.num_chains == q.num_chains
