"""Rough disk flux for craters of every kind of size beside a warp's 32 lanes, against
the restatement of the Observe stage (1e-12 of the step's flux: the same terms in
another order of summation), and no slower for few sub-facets than for many."""
import math
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WL = (4.6028, 11.0984, 22.6405)


def _case(ctx, nf, ntau, nsf):
    from binarytpm_gb300 import lib, mesh, problem

    v, f = mesh.perturbed_body(3, 0.39, 0.1, 1)
    f = f[:nf]
    prob = problem.Problem(v, f.astype(np.int32), *problem.empty_lists(nf), ntau=ntau, nx=8)
    s = lib.Solve(ctx, prob, precision=lib.REFERENCE)
    rng = np.random.default_rng(nsf)
    cv = rng.normal(size=(60, 3)).astype(np.float32)
    cf = ((np.arange(nsf)[:, None] + [0, 1, 2]) % 60).astype(np.int32)
    t = rng.uniform(80.0, 400.0, (nf, ntau, nsf)).astype(np.float32)
    seen = np.clip(rng.uniform(-0.4, 1.0, (nf, ntau, nsf)), 0.0, 1.0).astype(np.float32)
    warm, lit = lib.Crater(ctx, nf, ntau, 8, nsf), lib.Crater(ctx, nf, ntau, 0, nsf)
    warm.set_temperatures(t)
    lit.set_array(lib.Crater.SFC_SHADOW, seen)
    return prob, s, warm, lit, cv, cf, t, seen


@pytest.mark.parametrize("nf,nsf", [(1, 1), (37, 4), (300, 31), (300, 32), (257, 33), (70, 100), (70, 128)])
def test_crater_sizes(gpu_ctx, nf, nsf):
    from oracle import flux

    prob, s, warm, lit, cv, cf, t, seen = _case(gpu_ctx, nf, 3, nsf)
    observer = (0.9, 0.1, 0.3)
    got = s.disk_flux_rough(warm, lit, cv, cf, observer, WL)
    want = flux.rough_disk_flux(prob.vertices, prob.facets, 3, prob.pole, prob.polar, observer, 0.9, t.transpose(0, 2, 1),
                                seen.transpose(0, 2, 1), cv, cf, None, WL)
    assert np.all(np.abs(got - want) <= 1e-12 * np.abs(want).max(axis=0, keepdims=True))
    for x in (s, warm, lit):
        x.close()


def test_few_sub_facets_take_less_time(gpu_ctx):
    took = {}
    for nsf in (4, 32):
        _, s, warm, lit, cv, cf, _, _ = _case(gpu_ctx, 1280, 300, nsf)
        times = []
        for _ in range(5):
            t0 = time.perf_counter()
            s.disk_flux_rough(warm, lit, cv, cf, (0.9, 0.1, 0.3), WL)
            times.append(time.perf_counter() - t0)
        took[nsf] = min(times)
        for x in (s, warm, lit):
            x.close()
    assert took[4] < 0.7 * took[32], took
