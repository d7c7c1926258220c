"""The culled shadow drivers decide in 32 bits what lies clear of a decision and
leave the rest to the exact test: same flags as the plain drivers for metre-sized
and very large bodies, near and far observers, remainders of the 32-step windows,
and facets that share edges, planes and midpoints' lines of sight with others."""
import dataclasses
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _flags(ctx, prob, cull, precision):
    from binarytpm_gb300 import lib

    os.environ["ATPM_SHADOW_CULL"] = "1" if cull else "0"
    try:
        s = lib.Solve(ctx, prob, precision=precision)
        s.geometry_shadow()
        out = s.shadow(), s.cosillum()
        s.close()
    finally:
        os.environ.pop("ATPM_SHADOW_CULL", None)
    return out


def _binary(ctx, ntau, scale, shadowing, polar):
    from binarytpm_gb300 import workloads

    prob = workloads.binary_problem(ctx, p_subdiv=3, s_subdiv=2, ntau=ntau)
    return dataclasses.replace(prob, vertices=prob.vertices * scale, shadowing=shadowing, polar=polar)


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("shadowing", [1, 2])
@pytest.mark.parametrize("ntau,scale,polar", [(33, 1e-3, (1.0, 0.0, 0.0)), (31, 1.0, (0.7, 0.3, 2.0)),
                                              (64, 300.0, (1.0, 0.0, 0.0)), (40, 1.0, (3e-7, 0.1, 0.4)),
                                              (40, 1.0, (3e-8, 0.1, 0.4)), (40, 1.0, (1e-8, 0.1, 0.4))])
def test_flags_equal_the_plain_drivers(gpu_ctx, precision, shadowing, ntau, scale, polar):
    prob = _binary(gpu_ctx, ntau, scale, shadowing, polar)
    (a, ca), (b, cb) = _flags(gpu_ctx, prob, True, precision), _flags(gpu_ctx, prob, False, precision)
    assert np.array_equal(a, b)
    assert np.array_equal(ca, cb)


@pytest.mark.parametrize("precision", [0, 2])
def test_coincident_and_aligned_facets(gpu_ctx, precision):
    """Stacked grids of triangles facing the Sun, shifted by nothing, whole
    cells, halves and hairs: rays through vertices, along edges, ties in distance."""
    from binarytpm_gb300 import problem

    y, z = np.meshgrid(np.arange(7) * 0.1, np.arange(7) * 0.1, indexing="ij")
    flat = np.stack([np.zeros_like(y), y, z], -1).reshape(-1, 3)
    tris = []
    for i in range(6):
        for j in range(6):
            a, b, c, d = 7 * i + j, 7 * i + j + 1, 7 * i + j + 7, 7 * i + j + 8
            tris += [(a, b, c), (b, d, c)]
    tris = np.array(tris)
    sheets, facets = [], []
    for k, (dx, dy) in enumerate([(0.0, 0.0), (0.0, 0.0), (0.05, 0.0), (0.1, 0.1), (0.15, 0.05), (0.2, 1e-6), (0.25, 1e-9),
                                  (1e-9, 0.3)]):
        sheets.append(flat + np.array([dx, dy, 0.0]))
        facets.append((tris if k % 2 else tris[:, ::-1]) + k * len(flat))
    v, f = np.concatenate(sheets), np.concatenate(facets).astype(np.int32)
    nf = len(f)
    ptr = (np.arange(nf + 1) * nf).astype(np.int32)
    prob = problem.Problem(v, f, ptr, np.tile(np.arange(nf), nf).astype(np.int32), np.full(nf * nf, 1e-6, np.float32),
                           ntau=48, nx=8, pole=(1.2, 0.3))
    for shadowing in (1, 2):
        prob = dataclasses.replace(prob, shadowing=shadowing)
        if shadowing == 1:  # lists without the facet itself
            keep = prob.dep_idx != np.repeat(np.arange(nf), np.diff(prob.dep_ptr))
            prob = dataclasses.replace(prob, dep_idx=prob.dep_idx[keep], dep_vf=prob.dep_vf[keep],
                                       dep_ptr=(np.arange(nf + 1) * (nf - 1)).astype(np.int32))
        a, b = _flags(gpu_ctx, prob, True, precision), _flags(gpu_ctx, prob, False, precision)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
        assert 0 < a[0].sum() < a[0].size
