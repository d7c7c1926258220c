"""What stays in the device's stream-ordered pool: a view-factor call keeps at most
half a gigabyte of its scratch, and a context that goes gives back what is unused."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

RESERVED, USED = 5, 7  # CU_MEMPOOL_ATTR_RESERVED_MEM_CURRENT, _USED_MEM_CURRENT


def _held(attribute):
    cu, pool, v = C.CDLL("libcuda.so.1"), C.c_void_p(), C.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert cu.cuMemPoolGetAttribute(pool, attribute, C.byref(v)) == 0
    return v.value


def test_viewfactors_and_contexts_give_back(gpu_ctx):
    from binarytpm_gb300 import lib, problem

    lib.Context(0).close()
    before, used = _held(RESERVED), _held(USED)
    ctx = lib.Context(0)
    v, f = problem.binary_mesh(5, 4, 2)  # 25,600 facets
    ptr, idx, _, _, _ = lib.viewfactors(ctx, v, f, refine=False)
    assert len(idx) > 10 * len(f)
    assert _held(USED) == used
    assert _held(RESERVED) <= before + (512 << 20) + (64 << 20)  # whole 32 MB granules
    s = lib.Solve(ctx, problem.Problem(v, f, *problem.empty_lists(len(f)), ntau=720, nx=8), precision=lib.FAST)
    s.close()
    assert _held(RESERVED) > before + (300 << 20)  # kept for the next solve
    ctx.close()
    assert _held(RESERVED) <= before + (64 << 20)
