"""New contexts while the process-wide tuning cache holds an entry for their N and table: the device's name, which
the entry is compared with, is asked for once per device (the query takes 4 to 40 ms), not by every context and
not with the cache locked. Needs a B200."""
import threading
import time

import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu

N, BINS = 233, 777


def _prepare_ms(n=N):
    """Milliseconds of a fresh context's first prepare."""
    p = T.default_params(num_segments=n, mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, num_curvature_steps=BINS,
                         num_chains=8, paths_to_generate=8, max_sub_chain=8, max_angle=0.05)
    with T.Context(p) as ctx:
        t0 = time.perf_counter()
        ctx.prepare(T.make_bc((0, 0, 0), (0, 0, 1), (0, 0, 15), (0, 0, 1), 30.0))
        ms = 1e3 * (time.perf_counter() - t0)
        ctx.launch()
        return ms, ctx.collect().kernel_shape


def test_new_contexts_do_not_query_the_device_again(tmp_path):
    import torch
    before = sorted(_prepare_ms()[0] for _ in range(9))[4]
    f = tmp_path / "tune.json"
    f.write_text('{"entries": [{"device": "%s", "n": %d, "bins": %d, "group": 8, "spl": 32, "warps": 16, '
                 '"path_segments_per_s": 1.0}]}' % (torch.cuda.get_device_name(0), N, BINS))
    T.tuning_cache_load(str(f))
    runs = [_prepare_ms() for _ in range(9)]
    assert {shape for _, shape in runs} == {8 << 8 | 32}
    assert sorted(ms for ms, _ in runs)[4] < before + 2.0, (before, runs)
    # contexts on four threads at once find the entry too
    got = []
    threads = [threading.Thread(target=lambda: got.append(_prepare_ms()[1])) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [8 << 8 | 32] * 4
