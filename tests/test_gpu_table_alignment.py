"""Tables that do not start on 16 bytes: every second one of a batch with an odd number of bins, and a caller's table for the
allocation-free pass. Needs a B200.

An experiment in a batch gives the bits that it gives alone in one, where its table is the first; a table moved by 8 bytes
gives the same bits."""
import ctypes as C

import numpy as np
import pytest

import twisty_b200 as T
from twisty_b200 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins", [255, 1777, 4097])
@pytest.mark.parametrize("N", [20, 66, 256, 700])
def test_batches_of_odd_tables(N, bins):
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.6 * S, 0.1 * S, 0), (1, 0, 0), S)
    base = dict(num_segments=N, mu=1.0, eps=0.0225, scatter=10.0, num_steps_int=2000, num_curvature_steps=bins, perturb_seed=8,
                num_chains=64, paths_to_generate=64 * 9, paths_to_skip=5, max_sub_chain=32, max_angle=0.05)
    with T.Context(T.default_params(**base)) as ctx:
        x = T.make_experiment(bc, N, 10.0, 0.0225, 64 * 9)
        run = ctx.run_batch([x] * 4)
        res, grad, _, _ = ctx.adjoint_batch([x] * 4)
        for i in range(4):
            ctx.update(experiment_id=i, bootstrap_seed=i)
            (alone,), g, _, _ = ctx.adjoint_batch([x])
            assert alone.total_paths == run[i].total_paths == 64 * 9
            assert alone.log10_weight == run[i].log10_weight == res[i].log10_weight
            assert np.array_equal(grad[i], g[0])


@pytest.mark.parametrize("bins", [513, 4096])
@pytest.mark.parametrize("N", [24, 64, 384])
def test_a_callers_table_may_start_on_8_bytes(N, bins):
    import torch
    S = 0.16 * N
    p = T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=bins,
                         perturb_seed=7, max_sub_chain=32, max_angle=0.1)
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.8 * S, 0, 0), (1, 0, 0), S)
    init = T.bootstrap_curve(p, bc)
    with T.Context(p) as ctx:
        lut, info = ctx.build_lut(np.float32(S) / np.float32(N))
    table = np.stack([lut, np.append(lut[1:] - lut[:-1], np.float32(0))], axis=1).astype(np.float32)
    d_segs = torch.from_numpy((init[1:] - init[:-1]).astype(np.float32)).cuda()
    d_result = torch.zeros(C.sizeof(_abi.NoAllocResult), dtype=torch.uint8, device="cuda")
    room = torch.zeros(bins + 2, 2, device="cuda")
    assert room.data_ptr() % 16 == 0
    got = []
    for first in (0, 1):
        room[first:first + bins] = torch.from_numpy(table).cuda()
        args = _abi.NoAllocArgs(
            table=room[first:].data_ptr(), bins=bins, min_curvature=info.min_curvature, max_curvature=info.max_curvature,
            curvature_step=info.curvature_step, init_segments=d_segs.data_ptr(), num_segments=N, arclength=S, absorption=0.0,
            seed=7, experiment_id=0, chain_offset=0, num_chains=256, paths=256 * 20, burn_in=5, max_sub_chain=32, max_angle=0.1,
            result=d_result.data_ptr())
        torch.cuda.synchronize()
        assert _abi.load().twisty_run_noalloc(C.byref(args), None) == _abi.OK
        torch.cuda.synchronize()
        got.append(_abi.NoAllocResult.from_buffer_copy(d_result.cpu().numpy().tobytes()))
    assert got[0].valid_paths == 256 * 20 and got[1].valid_paths == 256 * 20
    assert got[0].log10_weight == got[1].log10_weight and got[0].rel_std_error == got[1].rel_std_error
