"""The plain form's kernel at each number of lanes per chain (8, 16, 32 by the pass's chains, and the
long chains whose positions stay in global memory) against the CPU oracle's chains of the same
proposals, and its paths with segment weights that are zero, negative or past the table. Needs a B200.

Positions, bins and blends are the oracle's bit for bit. A path's log10 weight is the FP64 sum of N - 1
logs in the oracle and the log of a product here: they differ by the sum's rounding, at
most N 2^-53 |log10 w|, and by 1e-11 for the accumulators."""
import numpy as np
import pytest

import twisty_b200 as T
from twisty_b200 import _abi

pytestmark = pytest.mark.gpu
F32 = np.float32
PI = float(F32(np.pi))


def _run(oracle, N, chains, steps, burn, angle, edit=None):
    S = max(0.12 * N, 2.0)
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.55 * S, 0.1 * S, 0), (1, 0, 0), S)
    lut, meta = oracle.lut_f32(oracle.wparams(1.0, 0.01, 10.0, 0.0, 2000, 512), F32(S) / F32(N))
    if edit:
        lut = lut.copy()
        edit(lut)
    p = T.default_params(num_segments=N, form=T.FORM_PLAIN_FP32, perturb_seed=19, num_chains=chains, max_angle=angle,
                         paths_to_generate=chains * steps, paths_to_skip=burn, mu=1.0, eps=0.01, scatter=10.0,
                         num_steps_int=2000, num_curvature_steps=512, bootstrap_kind=2)
    init = T.bootstrap_curve(p, bc)
    with T.Context(p) as ctx:
        ctx.set_lut(lut, _abi.LutInfo(meta.min_k, meta.max_k, meta.step, meta.min_w, meta.max_w, meta.ds, lut.size))
        ctx.set_initial_curve(init)
        r = ctx.run(bc)
        got, valid = ctx.chain_results(r.num_chains)
    o = oracle.run_chains(init, N, S, lut, meta, seed=19, n_chains=chains, steps=steps, burn_in=burn, max_angle=angle,
                          want_paths=True)
    assert r.num_chains == chains and r.steps_per_chain == steps
    return got - r.log10_normalizer, valid, r, o


@pytest.mark.parametrize("N,chains,steps,burn", [(4, 14300, 2, 1), (10, 14209, 3, 5), (66, 14300, 3, 2),   # 8 lanes
                                                 (20, 7200, 5, 3), (150, 7111, 2, 2),                       # 16
                                                 (7, 33, 40, 9), (33, 1, 100, 0), (513, 1000, 3, 4),        # 32
                                                 (4800, 5, 2, 3), (4801, 5, 2, 3)])                         # shared, global
def test_plain_lanes_match_oracle(oracle, N, chains, steps, burn):
    got, valid, r, o = _run(oracle, N, chains, steps, burn, PI if N < 200 else 0.1)
    assert r.failed_paths == 0 and np.array_equal(valid, o["chain_valid"])
    want = o["chain_log10"]
    assert np.all(np.abs(got - want) <= N * 2.0 ** -53 * np.abs(want) + 1e-11)


@pytest.mark.parametrize("N,chains", [(10, 14300), (20, 7200), (66, 300)])
def test_plain_paths_through_bad_table_entries_match_oracle(oracle, N, chains):
    def edit(lut):
        lut[60:64] = 0.0       # log10 -inf: a weight of zero
        lut[100:104] = -1e-3   # log10 NaN: an invalid path

    got, valid, r, o = _run(oracle, N, chains, 6, 4, PI, edit)
    w = o["path_log10"].reshape(chains, 6)
    ok = o["path_valid"].reshape(chains, 6) == 1
    assert np.array_equal(valid, ok.sum(axis=1)) and r.failed_paths == chains * 6 - int(valid.sum())
    assert 0 < r.failed_paths < chains * 6 and np.any(np.isneginf(w[ok]))
    for i in range(chains):
        x = w[i, ok[i]]
        if x.size == 0:
            assert np.isneginf(got[i])
        elif np.isneginf(x[0]):
            # CombinedWeightValues_C scales by its first weight: by 10^inf here, and stays NaN
            assert np.isnan(got[i])
        else:
            want = x.max() + np.log10(np.sum(10.0 ** (x - x.max())))
            assert abs(got[i] - want) <= N * 2.0 ** -53 * abs(want) + 1e-11
