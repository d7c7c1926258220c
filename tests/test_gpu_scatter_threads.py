"""Scattering of shapes and craters of different sizes on several host threads at
once, a handle each: every call succeeds with the result it has alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = 800


def _together(calls):
    """Runs each call CALLS times on a thread of its own."""
    failures, gate = [], threading.Barrier(len(calls))

    def work(call):
        gate.wait()
        try:
            for _ in range(CALLS):
                call()
        except Exception as e:  # noqa: BLE001
            failures.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


@pytest.mark.parametrize("precision", [0, 1])
def test_solves(gpu_ctx, precision):
    from binarytpm_gb300 import lib, problem

    solves = []
    for nf in (40, 900, 2600):  # 8 steps a CTA in both precisions
        rng = np.random.default_rng(nf)
        ptr = (2 * np.arange(nf + 1)).astype(np.int32)
        idx = np.sort((np.arange(nf)[:, None] + [1, 7]) % nf, axis=1).reshape(-1).astype(np.int32)
        facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
        prob = problem.Problem(rng.normal(size=(nf + 2, 3)), facets, ptr, idx, np.full(2 * nf, 0.05, np.float32),
                               ntau=16, nx=8, shadowing=0, albedo=0.3)
        s = lib.Solve(gpu_ctx, prob, precision=precision)
        s.geometry_shadow()
        s.scattering()
        solves.append((s, s.illumination()))
    _together([s.scattering for s, _ in solves])
    for s, want in solves:
        assert np.array_equal(s.illumination(), want)
        s.close()


@pytest.mark.parametrize("precision", [0, 2])
def test_craters(gpu_ctx, precision):
    from binarytpm_gb300 import lib

    craters = []
    for nsf in (16, 100, 128):
        rng = np.random.default_rng(nsf)
        nf, ntau = 2, 8
        c = lib.Crater(gpu_ctx, nf, ntau, 8, nsf, precision)
        v = rng.normal(size=(64, 3)).astype(np.float32)
        f = ((np.arange(nsf)[:, None] + [0, 1, 2]) % 64).astype(np.int32)
        vf = (rng.random((nsf, nsf)) / nsf).astype(np.float32)
        c.set_surface(v, f, vf, 8136.0)
        c.set_properties(np.zeros(nf, np.uint8), np.full(nf, 0.2, np.float32), np.zeros(nf, np.float32))
        for which in (c.SFC_SHADOW, c.SFC_SUN_ANGLE, c.GLOBAL_ILLUMINATION, c.GLOBAL_HEATING):
            c.set_array(which, rng.random((nf, ntau, nsf)).astype(np.float32))

        def step(c=c):
            c.scattering(1367.0)
            c.inst_equilibrium()

        c.scattering(1367.0)
        craters.append((c, step, c.get_array(c.ILLUMINATION)))
        c.zero_temperatures()
    _together([step for _, step, _ in craters])
    for c, _, want in craters:
        assert np.array_equal(c.get_array(c.ILLUMINATION), want)
        c.close()
