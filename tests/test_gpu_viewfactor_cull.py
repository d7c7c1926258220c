"""The occlusion culling's direction test in front of the exact one, and the
device's compaction and photon vectors: the lists of a float32 restatement that
puts every pair through the test, for rough, nested, touching, distant and
far-from-origin bodies and candidate counts around the block's spans."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dot(a, b):
    return (a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1]) + a[..., 2] * b[..., 2]


def _cross(a, b):
    return np.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1], a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                     a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def _lists(v, f):
    """3905/Shape_Selfheating/main.cpp:187-368 and 653-665 in float32."""
    v = v.astype(np.float32)
    v0, v1, v2 = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
    mid = ((v0 + v1) + v2) / np.float32(3.0)
    n = _cross(v1 - v0, v2 - v0)
    rows = []
    with np.errstate(all="ignore"):
        for G in range(len(f)):
            s = mid - mid[G]
            ok = (_dot(n[G], s) >= 0) & (_dot(-n, s) >= 0)
            ok[G] = False
            c = np.flatnonzero(ok)
            gv = mid[G] - mid[c]
            gl = np.sqrt(_dot(gv, gv))
            hidden = np.zeros(len(c), bool)
            for S in c:
                sv = mid[S] - mid[c]
                t = _dot(sv, n[S]) / _dot(gv, n[S])
                x = t[:, None] * gv + mid[c]
                q = [_dot(_cross(e, x - p), n[S]) >= 0
                     for e, p in ((v1[S] - v0[S], v0[S]), (-(v2[S] - v0[S]), v2[S]), (v2[S] - v1[S], v1[S]))]
                hidden |= (c != S) & (gl > np.sqrt(_dot(sv, sv))) & (t > 0) & q[0] & q[1] & q[2]
            rows.append(c[~hidden])
    return rows


def _shape(name):
    from binarytpm_gb300 import mesh

    if name == "rough":
        return mesh.grf_body(2, 0.39, 0.3, 0.4, 3)
    if name == "touching":
        return mesh.binary_system(mesh.grf_body(2, 0.39, 0.1, 0.5, 1), mesh.grf_body(2, 0.3, 0.1, 0.5, 2), 0.65)
    if name == "distant":
        return mesh.binary_system(mesh.perturbed_body(2, 0.39, 0.1, 1), mesh.perturbed_body(1, 0.05, 0.1, 2), 25.0)
    if name == "offset":
        v, f = mesh.grf_body(2, 0.39, 0.3, 0.4, 5)
        return v + np.array([20.0, -7.0, 3.0]), f
    inner, outer = mesh.perturbed_body(1, 0.1, 0.2, 6), mesh.perturbed_body(2, 1.0, 0.1, 7)
    return mesh.binary_system((outer[0], outer[1][:, [0, 2, 1]]), inner, 0.2)  # a body inside a hollow one


@pytest.mark.parametrize("name", ["rough", "touching", "distant", "offset", "nested"])
def test_lists_are_those_of_every_pair(gpu_ctx, name):
    from binarytpm_gb300 import lib

    v, f = _shape(name)
    ptr, idx, vf, vec, photo = lib.viewfactors(gpu_ctx, v, f, refine=False)
    want = _lists(v, f)
    assert np.array_equal(ptr, np.concatenate([[0], np.cumsum([len(r) for r in want])]))
    assert np.array_equal(idx, np.concatenate(want))
    # photon vectors: the rows' vectors over the facet's area, summed in list order
    v32 = v.astype(np.float32)
    n = _cross(v32[f[:, 1]] - v32[f[:, 0]], v32[f[:, 2]] - v32[f[:, 0]])
    area = np.sqrt(_dot(n, n)) / np.float32(2.0)
    for i in range(len(f)):
        t = np.zeros(3, np.float32)
        for k in range(ptr[i], ptr[i + 1]):
            t = t + vec[k] / area[i]
        assert np.array_equal(t, photo[i])
