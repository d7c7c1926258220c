"""Sums over view-factor lists of step rows (atpm_gather.cuh): single scattering,
FAST multiple scattering and the self-heating flux against the same sums in list
order in numpy, at one and at four (two in 64 bits) steps a lane, with lists of
lengths around the rows in flight (4, 8) and the entries a warp reads (32), and
step counts that are no multiple of a lane's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = (0, 1, 3, 4, 5, 7, 8, 9, 31, 32, 33, 63, 65)
SIZES = [(40, 1), (70, 6), (33, 129), (2003, 1237)]  # the last: 2,457 tiles of 32 x 32, the wide lanes


def _problem(nf, ntau, multiple):
    from binarytpm_gb300 import problem

    rng = np.random.default_rng(nf + ntau)
    n = np.minimum([LENGTHS[f % len(LENGTHS)] for f in range(nf)], nf - 1)
    ptr = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    rows = [np.sort(rng.choice(np.delete(np.arange(nf), f), k, replace=False)) for f, k in enumerate(n)]
    v = rng.normal(size=(nf + 2, 3))
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    return problem.Problem(v, facets, ptr, np.concatenate(rows).astype(np.int32),
                           rng.uniform(0.0, 0.01, ptr[-1]).astype(np.float32), ntau=ntau, nx=8, shadowing=0,
                           albedo=0.3, multiple_scattering=multiple)


def _sums(prob, start, rows, coefficient):
    """start + sum of coefficient(view factor) x the listed facet's row, in list order"""
    out = start.copy()
    for f in range(prob.nf):
        for k in range(prob.dep_ptr[f], prob.dep_ptr[f + 1]):
            out[f] = out[f] + coefficient(prob.dep_vf[k]) * rows[prob.dep_idx[k]]
    return out


@pytest.mark.parametrize("nf,ntau", SIZES)
@pytest.mark.parametrize("precision", ["reference", "fp64", "fast"])
def test_single_scattering_and_selfheating(gpu_ctx, nf, ntau, precision):
    from binarytpm_gb300 import lib
    from oracle import oracle

    prob = _problem(nf, ntau, 0)
    real = np.float64 if precision == "fp64" else np.float32
    s = lib.Solve(gpu_ctx, prob, precision=lib.PRECISIONS[precision])
    s.geometry_shadow()
    s.scattering()
    solar, alb = real(s.solar()), real(np.float32(prob.albedo) if real == np.float32 else prob.albedo)
    lit = s.cosillum().astype(real) * s.shadow().astype(real)
    got = s.illumination()
    want = _sums(prob, solar * lit, lit, lambda v: (real(v) * solar) * alb)
    if precision == "reference":
        assert np.array_equal(got, want)
    else:  # FAST: up to 66 terms of one sign, each within 2^-23; FP64: cosines read back in 32 bits
        assert np.all(np.abs(got - want) <= 2.0 ** (-22 if precision == "fp64" else -16) * np.abs(want))
    if precision == "fast":  # its self-heating goes over the tensor-core tiles
        s.close()
        return
    s.set_thermal_inertia(200.0)
    s.initialise_temperatures()
    t = (s.surface_temperature64() if precision == "fp64" else s.surface_temperature()[0]).astype(real)
    es = real(0.9) * real(5.67e-8)
    w = es * (t ** 4 if precision == "fp64" else oracle.glibc_powf(t.ravel(), 4.0).reshape(t.shape))
    q = s.selfheating_flux().T
    want = _sums(prob, np.zeros_like(w), w, lambda v: real(v))
    if precision == "reference":
        assert np.array_equal(q, want)
    else:  # returned in 32 bits; sigma and the emissivity may be the 32-bit constants
        assert np.all(np.abs(q - want) <= 2.0 ** -22 * np.abs(want))
    s.close()


@pytest.mark.parametrize("nf,ntau", SIZES)
def test_fast_multiple_scattering(gpu_ctx, nf, ntau):
    """FAST's Jacobi iterates and FP64's Gauss-Seidel ones end within
    accuracy x r / (1 - r) of the fixed point, r = albedo x the largest row sum
    (0.3 x 0.65 = 0.195); FAST rounds 66 terms in 32 bits."""
    from binarytpm_gb300 import lib

    prob = _problem(nf, ntau, 1)
    out = []
    for precision in (lib.FAST, lib.FP64):
        s = lib.Solve(gpu_ctx, prob, precision=precision)
        s.geometry_shadow()
        s.scattering()
        out.append(s.illumination().astype(np.float64))
        s.close()
    bound = 2 * prob.scattering_accuracy * 0.25 / prob.albedo + 2.0 ** -16 * np.abs(out[1])
    assert np.all(np.abs(out[0] - out[1]) <= bound)


@pytest.mark.parametrize("nf,ntau", [(40, 14), (301, 129), (515, 258)])
@pytest.mark.parametrize("min_entries,bound", [(8192, 2.0 ** -17), (8, 2.0 ** -14)])
def test_remainder_rows(gpu_ctx, monkeypatch, nf, ntau, min_entries, bound):
    """FAST self-heating with every entry in the sparse remainder (66 FP32
    products of one sign) and split between tiles and remainder (W in two BF16
    parts, 2^-17, and the tensor core's truncated sums, 66 of 2^-21); the view
    factors are exact in BF16."""
    from binarytpm_gb300 import lib

    monkeypatch.setenv("ATPM_TC_MIN_ENTRIES", str(min_entries))
    prob = _problem(nf, ntau, 0)
    prob.dep_vf[:] = np.ceil(prob.dep_vf * 2.0 ** 14) / np.float32(2.0 ** 14)
    rng = np.random.default_rng(ntau)
    s = lib.Solve(gpu_ctx, prob, precision=lib.FAST)
    s.set_forcing(rng.integers(0, 2, (nf, ntau)).astype(np.int32), (600 * rng.random((nf, ntau))).astype(np.float32))
    s.set_thermal_inertia(200.0)
    s.initialise_temperatures()
    s.revolution(0)
    t = s.surface_temperature64()
    q = s.selfheating_flux().T
    w = 0.9 * 5.67e-8 * t ** 4
    want = _sums(prob, np.zeros_like(w), w, float)
    assert np.all(np.abs(q - want) <= bound * want)
    s.close()
