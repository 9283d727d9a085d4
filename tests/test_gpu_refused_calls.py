"""A call that is refused after it has enqueued work returns with none of it in flight: the caller's arrays are its own
again. Needs a B200."""
import time

import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu


def test_a_refused_reweighing_leaves_no_copy_in_flight():
    import torch
    N, P = 256, 1 << 16
    S = 0.12 * N
    bc = T.make_bc((0, 0, 0), (1, 0, 0), (0.6 * S, 0.1, 0), (1, 0, 0), S)
    pinned = torch.zeros(P, N + 1, 3).pin_memory()       # 202 MB: 3 ms and more over the link
    with T.Context(T.default_params(num_segments=N, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=1024,
                                    paths_to_generate=1000)) as ctx:
        ctx.weight_paths(bc, np.zeros((4, N + 1, 3), np.float32))
        torch.cuda.synchronize()
        with pytest.raises(T.TwistyError) as e:
            ctx.weight_paths(bc, pinned.numpy(), form=T.FORM_FP64)
        t0 = time.perf_counter()
        torch.cuda.synchronize()
        left = time.perf_counter() - t0
        assert e.value.status == 8
    assert left < 1e-3, left
