"""Disk flux at facet, step and wavelength counts around the block, the flag
transpose's tiles and the wavelength limit, against the numpy restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("facets,ntau,nwl", [(1, 1, 1), (31, 33, 8), (255, 32, 3), (257, 31, 2), (320, 65, 5)])
@pytest.mark.parametrize("flags", [False, True])
def test_disk_flux_sizes(gpu_ctx, facets, ntau, nwl, flags):
    from binarytpm_gb300 import lib, mesh, problem
    from oracle import flux

    v, f = mesh.perturbed_body(2, 0.39, 0.1, 7)
    f = f[:facets].astype(np.int32)
    prob = problem.Problem(v, f, *problem.empty_lists(facets), ntau=ntau, nx=8, pole=(1.3, 0.2))
    rng = np.random.default_rng(facets)
    s = lib.Solve(gpu_ctx, prob, precision=lib.REFERENCE, revcap=2)
    s.set_forcing(np.ones((facets, ntau), np.int32), rng.uniform(1.0, 1300.0, (facets, ntau)).astype(np.float32))
    s.set_thermal_inertia(0.0)
    s.run()
    t = s.surface_temperature()[0].astype(np.float64)
    wl = tuple(rng.uniform(3.0, 30.0, nwl))
    vis = (rng.random((facets, ntau)) < 0.7).astype(np.int32) * 5 if flags else None
    obs = (0.9, 0.1, 0.3)
    got = s.disk_flux(obs, wl, vis)
    want = flux.disk_flux(v, f, ntau, prob.pole, prob.polar, obs, prob.emissivity, t.T, vis, wl)
    assert got.shape == want.shape == (ntau, nwl)
    # 1e-12 of the step's flux were every facet seen: sums run in another order
    scale = np.maximum(np.abs(want).max(axis=0, keepdims=True), 1e-300)
    assert np.all(np.abs(got - want) <= 1e-12 * scale)
    s.close()
