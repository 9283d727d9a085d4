"""Contexts on threads of their own, launching the same kernels with different amounts of shared memory: a launch must not
be refused for what another thread's launch needs. Needs a B200."""
import threading

import numpy as np
import pytest

import twisty_b200 as T

pytestmark = pytest.mark.gpu

BASE = dict(mu=1.0, eps=0.01, scatter=10.0, num_steps_int=2000, max_sub_chain=32, max_angle=0.05, perturb_seed=3, paths_to_skip=0)


def _bc(N):
    S = 0.12 * N
    return T.make_bc((0, 0, 0), (1, 0, 0), (0.6 * S, 0.1, 0), (1, 0, 0), S)


def _single(N, form, bins):
    p = T.default_params(num_segments=N, form=form, num_curvature_steps=bins, num_chains=8, paths_to_generate=8, **BASE)
    with T.Context(p) as ctx:
        ctx.prepare(_bc(N))
        ctx.launch()
        first = ctx.collect().log10_weight
        yield
        for i in range(1500):
            ctx.launch()
            if i % 100 == 99:
                assert ctx.collect().log10_weight == first


def _batch(N, bins):
    p = T.default_params(num_segments=N, num_curvature_steps=bins, num_chains=8, paths_to_generate=0, **BASE)
    exps = [T.make_experiment(_bc(N), N, 10.0, 0.01, 8)]
    with T.Context(p) as ctx:
        first = (ctx.run_batch(exps)[0].log10_weight, ctx.adjoint_batch(exps)[1].tolist())
        yield
        for _ in range(100):
            assert (ctx.run_batch(exps)[0].log10_weight, ctx.adjoint_batch(exps)[1].tolist()) == first


@pytest.mark.parametrize("jobs", [
    lambda: [_single(4700, T.FORM_PLAIN_FP32, 512), _single(40, T.FORM_PLAIN_FP32, 512)],
    lambda: [_single(256, T.FORM_COMPENSATED, 8192), _single(256, T.FORM_COMPENSATED, 512)],
    lambda: [_batch(256, 8192), _batch(256, 512)],
], ids=["plain", "compensated", "batch"])
def test_threads_with_different_shared_memory(jobs):
    errors = []
    start = threading.Barrier(2)

    def work(job):
        try:
            next(job)
            start.wait(60)
            for _ in job:
                pass
        except Exception as e:   # reported by the test's thread
            errors.append(repr(e))
            start.abort()

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs()]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
