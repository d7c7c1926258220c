"""Every form of the FAST depth sweep against every other, bit for bit.  Up to 56
advancing facets an SM the lane-split sweep takes a revolution, so the thread-per-
facet forms (three register budgets and the paired sweep; facet range or list of
active facets) run either with that sweep off or with more facets than the line:
facets of constant flux start in equilibrium and freeze at the first convergence
test, the others go on, so their share picks the form."""
import numpy as np
import pytest

from conftest import golden

pytestmark = pytest.mark.gpu


def _state(solve):
    return solve.surface_temperature64(), solve.depth_temperature(), solve.converged()


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("ntau,nx", [(48, 8), (720, 56)])
def test_variants_without_the_lane_split_sweep(gpu_ctx, monkeypatch, ntau, nx):
    """To convergence, with self-heating: pairs with one frozen facet among them."""
    from binarytpm_gb300 import lib

    prob = golden("binary_s3s1")[0].with_(ntau=ntau, nx=nx)
    first = lib.Solve(gpu_ctx, prob, precision=lib.FAST)
    first.geometry_shadow()
    first.scattering()
    solves = [first, first.clone()]
    monkeypatch.setenv("ATPM_AUTOTUNE", "0")

    def run():
        for s, ti in zip(solves, (60.0, 300.0)):
            s.set_thermal_inertia(ti)
            s.initialise_temperatures()
        counts = lib.batch_run(solves)
        return counts, [_state(s) for s in solves]

    want = run()  # the lane-split sweep
    assert any(0 < n < prob.nf for n in want[0][0])
    monkeypatch.setenv("ATPM_WARP_TAIL", "0")
    for variant in "1234":
        monkeypatch.setenv("ATPM_COND_VARIANT", variant)
        counts, states = run()
        assert first.last_run_config()[0] == int(variant)
        assert all(np.array_equal(a, b) for a, b in zip(counts, want[0]))
        assert all(_same(a, b) for a, b in zip(states, want[1]))
    for s in solves:
        s.close()


@pytest.mark.parametrize("frozen", [0.0, 0.05, 0.3, 0.55])
@pytest.mark.parametrize("odd", [0, 1])
def test_more_facets_than_the_line(gpu_ctx, monkeypatch, frozen, odd):
    """All or nearly all facets active (paired sweep, split pairs to the scalar one),
    most (scalar, facet range), and less than half (the list of active facets)."""
    import torch

    from binarytpm_gb300 import lib, problem

    line = 56 * torch.cuda.get_device_properties(0).multi_processor_count
    nf, ntau = int((line + 600) / (1.0 - frozen)) // 2 * 2 + odd, 48
    rng = np.random.default_rng(int(100 * frozen))
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    prob = problem.Problem(rng.normal(size=(nf + 2, 3)), facets, *problem.empty_lists(nf), ntau=ntau, nx=8)
    steady = rng.random(nf) < frozen
    flux = np.where(steady[:, None], 400.0, 900.0 * rng.random((nf, ntau))).astype(np.float32)
    s = lib.Solve(gpu_ctx, prob, precision=lib.FAST, revcap=10)
    s.set_forcing(np.ones((nf, ntau), np.int32), flux)
    monkeypatch.setenv("ATPM_AUTOTUNE", "0")
    got = []
    for tail, variant in [("0", "1"), ("1", "1"), ("1", "2"), ("1", "3"), ("1", "4"), ("0", "4")]:
        monkeypatch.setenv("ATPM_WARP_TAIL", tail)
        monkeypatch.setenv("ATPM_COND_VARIANT", variant)
        s.set_thermal_inertia(400.0)
        s.initialise_temperatures()
        counts = s.run()
        # the forms this case is for: revolutions 7 to 9 begin with these facets active
        active = nf - counts[6:9]
        assert len(counts) == 10 and (active > line).all()
        assert ((2 * active <= nf) == (frozen > 0.5)).all() and ((active >= 0.9 * nf) == (frozen < 0.1)).all()
        got.append((counts,) + _state(s))
    assert all(_same(g, got[0]) for g in got[1:])
    s.close()
