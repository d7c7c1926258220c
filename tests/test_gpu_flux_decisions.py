"""Disk flux beside its decisions: a facet (or a crater's sub-facet) that faces the
observer squarely counts or not as the stage's own arithmetic has it (its acos is
NaN where the cosine rounds above 1), a facet seen exactly edge-on keeps its crater's
light, and an observer near the body sees positions rounded as the stage rounds them.
The bar is that of the plain comparison, 1e-12 of the step's flux (the same terms in
another order of summation)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WL = (4.6028, 11.0984, 22.6405)
POLAR = (1e-6, 0.0, 0.0)  # so near that the heliocentric positions keep the normals' direction
POLE = (math.pi / 2, 0.0)


def _solve(ctx, normals, polar, size=1.0, shift=None):
    """A triangle of each normal, its midpoint at the body's centre (or `shift`)."""
    from binarytpm_gb300 import lib, problem

    nf = len(normals)
    other = np.where(np.abs(normals[:, :1]) < 0.9, [[1.0, 0.0, 0.0]], [[0.0, 1.0, 0.0]])
    a = np.cross(other, normals)
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b = np.cross(normals, a)
    v = size * np.stack([-(a + b), a, b], 1).reshape(-1, 3)
    if shift is not None:
        v = v + np.repeat(shift, 3, axis=0)
    prob = problem.Problem(v, np.arange(3 * nf, dtype=np.int32).reshape(-1, 3), *problem.empty_lists(nf), ntau=1, nx=8,
                           polar=polar, pole=POLE)
    s = lib.Solve(ctx, prob, precision=lib.REFERENCE)
    s.set_forcing(np.ones((nf, 1), np.int32), np.linspace(200.0, 900.0, nf, dtype=np.float32)[:, None])
    s.set_thermal_inertia(100.0)
    s.initialise_temperatures()
    return prob, s


def _toward(direction, distance):
    """The geocentric position whose observer lies in `direction` from the body."""
    x, y, z = -direction
    return distance, math.asin(z), math.atan2(y, x)


def _close(got, want):
    assert np.all(np.abs(got - want) <= 1e-12 * np.abs(want).max()), np.max(np.abs(got - want)) / np.abs(want).max()


def _directions(n, seed):
    d = np.random.default_rng(seed).normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def test_facets_that_face_the_observer(gpu_ctx):
    from oracle import flux

    normals = _directions(96, 1)
    normals[:3] = np.eye(3)
    prob, s = _solve(gpu_ctx, normals, POLAR)
    temps = s.surface_temperature()[0].astype(np.float64)
    for n in normals:
        observer = _toward(n, POLAR[0])
        _close(s.disk_flux(observer, WL),
               flux.disk_flux(prob.vertices, prob.facets, 1, POLE, POLAR, observer, 0.9, temps.T, None, WL))
    s.close()


@pytest.mark.parametrize("distance", [1.0, 1e-4, 1e-7])
def test_observers_near_a_body_far_from_the_origin(gpu_ctx, distance):
    from oracle import flux

    normals = _directions(200, 2)
    prob, s = _solve(gpu_ctx, normals, (1.0, 0.1, 0.4), 40.0, np.random.default_rng(3).normal(size=(200, 3)) * 900.0)
    temps = s.surface_temperature()[0].astype(np.float64)
    for n in normals[:8]:
        observer = _toward(n, distance)
        _close(s.disk_flux(observer, WL), flux.disk_flux(prob.vertices, prob.facets, 1, POLE, (1.0, 0.1, 0.4), observer,
                                                         0.9, temps.T, None, WL))
    s.close()


def test_craters_of_facets_squarely_seen_and_edge_on(gpu_ctx):
    from binarytpm_gb300 import lib
    from oracle import flux

    normals = np.concatenate([np.eye(3), -np.eye(3), _directions(40, 4)])
    nf = len(normals)
    prob, s = _solve(gpu_ctx, normals, POLAR)
    # a flat floor and three sides
    cv = np.array([(0, 0, 0), (1, 0, 0), (0, 1, 0), (2, 0, 1), (0, 2, 1), (-1, -1, 1)], np.float32)
    cf = np.array([(0, 1, 2), (1, 3, 2), (0, 2, 5), (0, 5, 1)], np.int32)
    rng = np.random.default_rng(5)
    t = rng.uniform(100.0, 400.0, (nf, 1, 4)).astype(np.float32)
    seen = rng.uniform(0.1, 1.0, (nf, 1, 4)).astype(np.float32)
    warm = lib.Crater(gpu_ctx, nf, 1, 8, 4)
    warm.set_temperatures(t)
    lit = lib.Crater(gpu_ctx, nf, 1, 0, 4)
    lit.set_array(lib.Crater.SFC_SHADOW, seen)
    for n in normals:
        observer = _toward(n, POLAR[0])
        want = flux.rough_disk_flux(prob.vertices, prob.facets, 1, POLE, POLAR, observer, 0.9, t.transpose(0, 2, 1),
                                    seen.transpose(0, 2, 1), cv, cf, None, WL)
        _close(s.disk_flux_rough(warm, lit, cv, cf, observer, WL), want)
    warm.close()
    lit.close()
    s.close()
