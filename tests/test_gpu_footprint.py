"""atpm_solve_footprint against the device memory that a solve and its setup take
at their peak, from the stream-ordered pool's own high-water mark."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

USED_NOW, USED_HIGH = 7, 8  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT, _HIGH


def _pool():
    cu, pool = C.CDLL("libcuda.so.1"), C.c_void_p()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0

    def read(attribute):
        v = C.c_uint64()
        assert cu.cuMemPoolGetAttribute(pool, attribute, C.byref(v)) == 0
        return v.value

    def mark():
        assert cu.cuMemPoolSetAttribute(pool, USED_HIGH, C.byref(C.c_uint64(0))) == 0
        return read(USED_NOW)

    return mark, lambda: read(USED_HIGH)


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("shadowing,subdivisions,ntau", [(0, 4, 360), (1, 4, 360), (2, 3, 96), (2, 5, 360)])
@pytest.mark.parametrize("multiple", [0, 1])
def test_footprint_is_the_peak(gpu_ctx, precision, shadowing, subdivisions, ntau, multiple):
    from binarytpm_gb300 import lib, workloads

    prob = workloads.binary_problem(gpu_ctx, p_subdiv=subdivisions, s_subdiv=2, ntau=ntau).with_(
        shadowing=shadowing, multiple_scattering=multiple, nx=16)
    first = lib.Solve(gpu_ctx, prob, precision=precision)  # the shape's tiles are shared, not a solve's own
    mark, high = _pool()
    before = mark()
    s = first.clone()
    s.geometry_shadow()
    s.scattering()
    s.shadow()
    took, counted = high() - before, lib.footprint(prob, precision)
    slack = 96 << 20 if shadowing == 2 else 2 << 20  # a grid's cells depend on the shape; page rounding
    assert took <= counted <= 1.25 * took + slack, (took, counted)
    s.close()
    first.close()
