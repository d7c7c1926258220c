"""FAST batches of exactly as many revolutions as the autotuner times, and one
either side: the first batch of its kind, a later one and one that is not tuned
give the same revolutions, counts and temperatures."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("caps", [[4], [5], [6], [5, 5], [5, 5, 5], [5, 7, 5]])
def test_the_first_run_of_a_kind(gpu_ctx, monkeypatch, caps):
    from binarytpm_gb300 import lib, problem

    nf, ntau = 300, 48
    rng = np.random.default_rng(0)
    v = rng.normal(size=(nf + 2, 3))
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    prob = problem.Problem(v, facets, *problem.empty_lists(nf), ntau=ntau, nx=8)
    flux = (600.0 * rng.random((nf, ntau))).astype(np.float32)
    ctx = lib.Context(0)  # nothing tuned yet
    got = []
    for tune in "110":
        monkeypatch.setenv("ATPM_AUTOTUNE", tune)
        solves = [lib.Solve(ctx, prob, precision=lib.FAST, revcap=c) for c in caps]
        for s in solves:
            s.set_forcing(np.ones((nf, ntau), np.int32), flux)
            s.set_thermal_inertia(40.0)
            s.initialise_temperatures()
        counts = lib.batch_run(solves)
        assert [len(c) for c in counts] == caps
        assert solves[0].last_run_stats()[0] > 0.0
        got.append((counts, [s.surface_temperature64() for s in solves]))
        for s in solves:
            s.close()
    for counts, temps in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(counts, got[0][0]))
        assert all(np.array_equal(a, b) for a, b in zip(temps, got[0][1]))
    ctx.close()
