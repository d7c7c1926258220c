"""Calls whose scratch memory only makes them faster, with device memory for less
than that: they go on without it, with the same results."""
import contextlib
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRANULE = 32 << 20  # a pool's limit is rounded up to whole ones


class _Location(C.Structure):
    _fields_ = [("type", C.c_int), ("id", C.c_int)]


class _PoolProps(C.Structure):  # CUmemPoolProps
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("location", _Location), ("security", C.c_void_p),
                ("max_size", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


@contextlib.contextmanager
def _room(size):
    """Device 0's stream-ordered allocations come from a pool with `size` bytes left."""
    cu = C.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, rc

    pool, before, filler = C.c_void_p(), C.c_void_p(), C.c_void_p()
    props = _PoolProps(1, 0, _Location(1, 0), None, GRANULE, 0)
    ok(cu.cuMemPoolCreate(C.byref(pool), C.byref(props)))
    ok(cu.cuMemAllocFromPoolAsync(C.byref(filler), C.c_size_t(GRANULE - size), pool, None))
    ok(cu.cuStreamSynchronize(None))
    ok(cu.cuDeviceGetMemPool(C.byref(before), 0))
    ok(cu.cuDeviceSetMemPool(0, pool))
    try:
        yield
    finally:
        ok(cu.cuDeviceSetMemPool(0, before))
        ok(cu.cuMemFreeAsync(filler, None))
        ok(cu.cuCtxSynchronize())
        ok(cu.cuMemPoolDestroy(pool))


def _problem(nf=80000, ntau=128, **kw):
    """Many facets over few vertices: whatever goes by facets and steps is large."""
    from binarytpm_gb300 import problem

    rng = np.random.default_rng(3)
    facets = np.stack([(np.arange(nf) * k + j) % 41 for j, k in enumerate((1, 3, 7))], 1).astype(np.int32)
    facets[:, 2] = np.where((facets[:, 2] == facets[:, 0]) | (facets[:, 2] == facets[:, 1]), (facets[:, 2] + 11) % 41,
                            facets[:, 2])
    near = np.sort(rng.integers(0, nf, (2000, 5)), axis=1)
    ptr = np.minimum(5 * np.arange(nf + 1), near.size).astype(np.int32)
    return problem.Problem(rng.normal(size=(41, 3)), facets, ptr, near.reshape(-1).astype(np.int32),
                           np.full(near.size, 0.05, np.float32), ntau=ntau, nx=8, **kw)


@pytest.mark.parametrize("precision", [0, 2])
def test_shadowing_without_window_boxes(gpu_ctx, precision):
    from binarytpm_gb300 import lib

    s = lib.Solve(gpu_ctx, _problem(), precision=precision)
    s.geometry_shadow()
    want = s.shadow()
    with _room(4 << 20):  # projected vertices fit, the boxes of 80,000 facets and 4 windows (5 MB) do not
        s.geometry_shadow()
    assert np.array_equal(s.shadow(), want)
    assert 0 < want[:2000].sum() < want[:2000].size
    s.close()


@pytest.mark.parametrize("nf,ntau", [(80000, 128), (70001, 127)])
def test_shadow_flags_without_staging(gpu_ctx, nf, ntau):
    from binarytpm_gb300 import lib

    s = lib.Solve(gpu_ctx, _problem(nf, ntau, shadowing=0), precision=0)
    s.geometry_shadow()
    want = s.shadow()
    with _room(4 << 20):
        got = s.shadow()
    assert np.array_equal(got, want)
    assert 0 < want.sum() < want.size
    s.close()


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_single_scattering_without_rows(gpu_ctx, precision):
    from binarytpm_gb300 import lib

    s = lib.Solve(gpu_ctx, _problem(shadowing=0, albedo=0.3, multiple_scattering=0), precision=precision)
    s.geometry_shadow()
    s.scattering()
    want = s.illumination()
    s.set_albedo(0.0)
    s.scattering()
    direct = s.illumination()
    s.set_albedo(0.3)
    with _room(4 << 20):
        s.scattering()
    got = s.illumination()
    nan = np.isnan(want)  # some facets here have two corners alike
    assert np.array_equal(np.isnan(got), nan)
    got, want, direct = got[~nan], want[~nan], direct[~nan]
    if precision == 2:  # FAST may contract its products either way: two roundings of terms below the sum
        assert np.all(np.abs(got - want) <= 8 * 2.0 ** -24 * np.abs(want) + 1e-30)
    else:
        assert np.array_equal(got, want)
    assert (want != direct).any()
    s.close()


@pytest.mark.parametrize("flags", [True, False])
def test_disk_flux_a_few_steps_at_a_time(gpu_ctx, flags):
    from binarytpm_gb300 import lib

    nf, ntau = 12000, 701
    prob = _problem(nf, ntau, shadowing=0)
    s = lib.Solve(gpu_ctx, prob, precision=0)
    rng = np.random.default_rng(8)
    s.set_forcing(np.ones((nf, ntau), np.int32), (600 * rng.random((nf, ntau))).astype(np.float32))
    s.set_thermal_inertia(100.0)
    s.initialise_temperatures()
    seen = (rng.random((nf, ntau)) < 0.7).astype(np.int32) if flags else None
    observer, wl = (0.9, 0.1, 0.3), (4.6, 11.1)
    want = s.disk_flux(observer, wl, seen)
    with _room(1 << 20):  # the block sums take 0.53 MB, the positions 0.69, the flags 42
        got = s.disk_flux(observer, wl, seen)
    assert np.array_equal(got, want)
    assert (want > 0).all()
    s.close()


def test_gauss_seidel_without_its_order(gpu_ctx):
    from binarytpm_gb300 import lib

    got = []
    for size in (GRANULE // 2, 1_900_000):  # the sweeps take 1.80 MB, the level order 0.23
        s = lib.Solve(gpu_ctx, _problem(50000, 1, shadowing=0, albedo=0.3), precision=0)
        s.geometry_shadow()
        with _room(size):
            s.scattering()
        got.append(s.illumination())
        s.close()
    assert np.array_equal(got[0], got[1], equal_nan=True)


@pytest.mark.parametrize("failing", ["scattering", "viewfactors"])
def test_a_failed_allocation_fails_one_call(gpu_ctx, failing):
    from binarytpm_gb300 import lib, problem

    s = lib.Solve(gpu_ctx, _problem(shadowing=0, albedo=0.3), precision=0)
    s.geometry_shadow()
    v, f = problem.binary_mesh(4, 3, 2)
    call = {"scattering": s.scattering, "viewfactors": lambda: lib.viewfactors(gpu_ctx, v, f)}[failing]
    with _room(256 << 10):
        with pytest.raises(lib.AtpmError):
            call()
    s.geometry_shadow()  # what failed is not found again by the next launches
    call()
    s.close()
