"""FAST products of few work items, dealt out by steps (k_prepare), against the
same solves in a batch too large for that, bit for bit: chunks of every number of
16-step groups, parts that do not divide them, row blocks without a tile, and
facets that freeze while others go on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,ntau,entries", [(130, 96, 20), (130, 17, 20), (300, 160, 40), (300, 161, 40),
                                             (700, 330, 60), (1500, 256, 30), (64, 200, 0)])
def test_parts_are_the_whole(gpu_ctx, monkeypatch, nf, ntau, entries):
    from binarytpm_gb300 import lib, problem

    monkeypatch.setenv("ATPM_TC_MIN_ENTRIES", "4")
    rng = np.random.default_rng(ntau)
    rows = [np.sort(rng.choice(nf, entries if f % 200 < 150 else 0, replace=False)) for f in range(nf)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    v = rng.normal(size=(nf + 2, 3))
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    prob = problem.Problem(v, facets, ptr, np.concatenate(rows).astype(np.int32),
                           rng.uniform(0.0, 0.2 / max(entries, 1), ptr[-1]).astype(np.float32), ntau=ntau, nx=8)
    flux = (600.0 * rng.random((nf, ntau))).astype(np.float32)
    first = lib.Solve(gpu_ctx, prob, precision=lib.FAST, revcap=14)
    first.set_forcing(np.ones((nf, ntau), np.int32), flux)
    many = [first] + [first.clone() for _ in range(39)]
    for s in many:
        s.set_thermal_inertia(40.0)
        s.initialise_temperatures()
    together = lib.batch_run(many)[0]
    want = first.surface_temperature64()
    first.set_thermal_inertia(40.0)
    first.initialise_temperatures()
    assert np.array_equal(together, first.run())
    assert np.array_equal(first.surface_temperature64(), want)
    for s in many:
        s.close()
