"""Every stage of solves and craters on several host threads at once, a handle each:
the results each has alone, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(ctx, seed):
    from binarytpm_gb300 import lib, mesh, problem

    rng = np.random.default_rng(seed)
    v, f = mesh.perturbed_body(int(rng.integers(1, 4)), 0.39, 0.2, seed)
    nf = len(f)
    idx = np.sort((np.arange(nf)[:, None] + rng.integers(1, nf, (1, 6))) % nf, axis=1)
    prob = problem.Problem(v, f.astype(np.int32), (6 * np.arange(nf + 1)).astype(np.int32),
                           idx.reshape(-1).astype(np.int32), np.full(6 * nf, 0.02, np.float32), ntau=48, nx=8, albedo=0.2)
    first = lib.Solve(ctx, prob, precision=seed % 3, revcap=9)
    first.geometry_shadow()
    first.scattering()
    solves = [first] + [first.clone() for _ in range(seed % 4)]
    for k, s in enumerate(solves):
        s.set_thermal_inertia(50.0 + 100.0 * k)
        s.initialise_temperatures()
    out = [first.shadow(), first.illumination()] + lib.batch_run(solves)
    for s in solves:
        out += [s.surface_temperature64(), s.selfheating_flux(), s.disk_flux((0.9, 0.1, 0.3), (5.0, 11.0))]
        s.close()
    return out


def _crater(ctx, seed):
    from binarytpm_gb300 import lib

    rng = np.random.default_rng(seed)
    nf, ntau, nsf = 1 + seed % 5, 40, 100
    c = lib.Crater(ctx, nf, ntau, 8, nsf, 2 * (seed % 2))
    v = rng.normal(size=(60, 3)).astype(np.float32)
    c.set_surface(v, ((np.arange(nsf)[:, None] + [0, 1, 2]) % 60).astype(np.int32),
                  (rng.random((nsf, nsf)) / nsf).astype(np.float32), 8136.0)
    c.set_properties(np.zeros(nf, np.uint8), np.full(nf, 0.1, np.float32), np.full(nf, 200.0, np.float32))
    c.set_array(c.SHADOW, np.ones((nf, ntau), np.int32))
    c.set_array(c.SUN_VECTOR, 1e3 * rng.normal(size=(nf, ntau, 3)))
    for which in (c.SFC_SHADOW, c.SFC_SUN_ANGLE, c.GLOBAL_ILLUMINATION, c.GLOBAL_HEATING):
        c.set_array(which, rng.random((nf, ntau, nsf)))
    c.partial_shadow()
    c.scattering(1367.0)
    c.initialise_temperatures()
    for _ in range(2):
        c.inertia_difference()
    out = [c.get_array(c.ILLUMINATION), *c.get_temperatures()]
    c.zero_temperatures()
    c.inst_equilibrium()
    out += [c.get_temperatures()[1]]
    c.close()
    return out


def test_all_stages_beside_each_other(gpu_ctx):
    jobs = [(_solve, s) for s in range(36)] + [(_crater, s) for s in range(12)]
    want = [call(gpu_ctx, seed) for call, seed in jobs]
    got, errors, lock, order = [None] * len(jobs), [], threading.Lock(), iter(range(len(jobs)))

    def work():
        while True:
            with lock:
                i = next(order, None)
            if i is None:
                return
            try:
                got[i] = jobs[i][0](gpu_ctx, jobs[i][1])
            except Exception as e:  # noqa: BLE001
                errors.append((i, e))

    threads = [threading.Thread(target=work) for _ in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for (call, seed), a, b in zip(jobs, want, got):
        assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b)), (call.__name__, seed)
