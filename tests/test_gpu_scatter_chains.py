"""Gauss-Seidel scattering of lists that chain facet to facet: the facet-by-facet
kernel takes them where the levels are many, with the same bits on both sides of
that line, and long chains take no longer than lists that cannot go by levels."""
import time

import numpy as np
import pytest

from test_gpu_scatter_levels import _check

pytestmark = pytest.mark.gpu


def _chain(nf, ntau, stride, ascending=True):
    from binarytpm_gb300 import problem

    rows = [[g for g in (f - stride, f + stride)[:: 1 if ascending else -1] if 0 <= g < nf] for f in range(nf)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    idx = np.concatenate(rows).astype(np.int32)
    rng = np.random.default_rng(nf)
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    return problem.Problem(rng.normal(size=(nf + 2, 3)), facets, ptr, idx,
                           rng.uniform(0.0, 0.2, len(idx)).astype(np.float32), ntau=ntau, nx=8, shadowing=0, albedo=0.3,
                           scattering_accuracy=1e-4)


@pytest.mark.parametrize("precision", ["reference", "fp64"])
@pytest.mark.parametrize("nf,ntau,stride", [(2, 5, 1), (301, 9, 1), (301, 9, 2), (7041, 7, 1), (7041, 7, 2)])
def test_chains(gpu_ctx, nf, ntau, stride, precision):
    _check(gpu_ctx, _chain(nf, ntau, stride), precision)


def test_long_chains_are_not_swept_by_levels(gpu_ctx):
    from binarytpm_gb300 import lib

    best = []
    for ascending in (True, False):  # unsorted lists have no level order
        s = lib.Solve(gpu_ctx, _chain(20480, 720, 1, ascending), precision=lib.REFERENCE)
        s.geometry_shadow()
        s.scattering()
        took = []
        for _ in range(4):
            t = time.perf_counter()
            s.scattering()
            took.append(time.perf_counter() - t)
        best.append(min(took))
        s.close()
    assert best[0] < 1.5 * best[1], best
