"""Batches of few experiments, whose items are split over smaller CTAs, against the same experiments in front of many
others, where they are not: the split moves chains between CTAs only, so every result has the same bits. Needs a
B200."""
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


def _exp(N, paths):
    S = max(0.12 * N, 1.0)
    return T.make_experiment(T.make_bc((0, 0, 0), (1, 0, 0), (0.55 * S, 0.1 * S, 0), (1, 0, 0), S), N, 10.0, 0.01, paths)


@pytest.mark.parametrize("sizes", [[(1024, 20000)], [(16, 3), (700, 1 << 14)], [(66, 1 << 14), (12, 5000), (300, 4097)],
                                   [(850, 1 << 13)] * 5, [(128, 1 << 17), (512, 1 << 15), (1000, 30000), (4, 100)]])
def test_split_items_keep_the_results(sizes):
    p = T.default_params(mu=1.0, num_steps_int=2000, num_curvature_steps=1024, paths_to_skip=16, perturb_seed=3, bootstrap_seed=11,
                         max_sub_chain=32, max_angle=0.1)
    few = [_exp(*s) for s in sizes]
    filler = [_exp(40 + i, 1 << 16) for i in range(300)]
    with T.Context(p) as ctx:
        a = ctx.run_batch(few)
    with T.Context(p) as ctx:
        b = ctx.run_batch(few + filler)
    for x, y, s in zip(a, b, sizes):
        assert x.total_paths == y.total_paths == s[1] and x.failed_paths == y.failed_paths == 0
        assert x.log10_weight == y.log10_weight and x.num_chains == y.num_chains
        assert x.rel_std_error == y.rel_std_error or s[1] < 6
