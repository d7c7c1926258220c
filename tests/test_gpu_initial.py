"""Initial temperatures (k_initial) against the restatement in step order: facet
counts around a block's 64, step counts around the 32 of a load and of a span,
and FAST's W, which the first revolution must find as the rebuild from the
surface temperatures leaves it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (63, 31), (64, 32), (65, 33), (130, 97), (1000, 45)]


def _solve(ctx, nf, ntau, precision):
    from binarytpm_gb300 import lib, problem

    rng = np.random.default_rng(nf)
    n = rng.integers(0, 12, nf) if nf > 12 else np.zeros(nf, int)
    ptr = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    idx = rng.integers(0, nf, ptr[-1]).astype(np.int32)
    v = rng.normal(size=(nf + 2, 3))
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    prob = problem.Problem(v, facets, ptr, idx, rng.uniform(0.0, 0.03, ptr[-1]).astype(np.float32), ntau=ntau, nx=8)
    flux = (1.0 + 600.0 * rng.random((nf, ntau))).astype(np.float32)
    s = lib.Solve(ctx, prob, precision=lib.PRECISIONS[precision])
    s.set_forcing(np.ones((nf, ntau), np.int32), flux)
    s.set_thermal_inertia(200.0)
    s.initialise_temperatures()
    return s, prob, flux


@pytest.mark.parametrize("nf,ntau", SIZES)
@pytest.mark.parametrize("precision", ["reference", "fp64", "fast"])
def test_initial_temperatures(gpu_ctx, nf, ntau, precision):
    from oracle import oracle

    s, prob, flux = _solve(gpu_ctx, nf, ntau, precision)
    real = np.float64 if precision == "fp64" else np.float32
    mean = np.zeros(nf, real)
    inv = real(1) / real(ntau)
    for step in range(ntau):
        mean = mean + inv * flux[:, step].astype(real)
    got = s.surface_temperature64()
    assert np.array_equal(got, np.repeat(got[:, :1], ntau, 1))
    depth = s.depth_temperature()
    assert np.array_equal(depth, np.repeat(got[:, :1], prob.nx + 1, 1).astype(np.float32))
    if precision == "reference":
        x = (np.float32(1) - np.float32(prob.albedo)) * mean / np.float32(0.9 * 5.67e-8)
        assert np.array_equal(got[:, 0], oracle.glibc_powf(x, 0.25))
    else:  # FAST: 97 fused additions and a 32-bit root; FP64: constants that may be 32-bit ones
        x = (1.0 - prob.albedo) * mean / (0.9 * 5.67e-8)
        assert np.all(np.abs(got[:, 0] - x ** 0.25) <= 2.0 ** -18 * x ** 0.25)
    s.close()


@pytest.mark.parametrize("nf,ntau", SIZES[1:])
@pytest.mark.parametrize("min_entries", [1, 8192])
def test_first_revolution_finds_w(gpu_ctx, monkeypatch, nf, ntau, min_entries):
    monkeypatch.setenv("ATPM_TC_MIN_ENTRIES", str(min_entries))
    out = []
    for rebuild in (False, True):
        s = _solve(gpu_ctx, nf, ntau, "fast")[0]
        if rebuild:
            s.selfheating_flux()
        s.revolution(0)
        out.append(s.surface_temperature64())
        s.close()
    assert np.array_equal(out[0], out[1])
