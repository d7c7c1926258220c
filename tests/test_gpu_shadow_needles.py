"""The culled shadow drivers on needles: long facets with one short edge seen so
nearly edge-on that the projected triangle's orientation drowns in 32-bit rounding.
Points inside them are the exact test's to decide: same flags as the plain drivers."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AU_KM = 149.6e6


def _needles(n, seed, distance):
    """n needles and, behind each, a small facet toward the Sun whose midpoint
    lies on the line through a point of the needle (heliocentric, body on the x axis)."""
    rng = np.random.default_rng(seed)
    along = rng.uniform(0, 2 * np.pi, n)
    u = np.stack([np.zeros(n), np.cos(along), np.sin(along)], 1)
    w = np.stack([np.zeros(n), -np.sin(along), np.cos(along)], 1)
    d = np.array([[1.0, 0.0, 0.0]])
    length = 10 ** rng.uniform(-0.7, 0.3, (n, 1))
    short = length / 10 ** rng.uniform(2.3, 4, (n, 1))
    v0 = np.concatenate([rng.uniform(-0.2, 0.2, (n, 1)), rng.uniform(-0.4, 0.4, (n, 2))], 1)
    v1 = v0 + length * u + rng.uniform(-1, 1, (n, 1)) * length * d
    a = rng.uniform(-1, 1, (n, 1))
    tilt = 10 ** rng.uniform(-9, -4, (n, 1)) * rng.choice([-1, 1], (n, 1))
    v2 = v1 + short * (a * u + (1 - np.abs(a)) * d + tilt * w)
    needles = np.stack([v0, v1, v2], 1)
    needles = np.take_along_axis(needles, (np.arange(3) + rng.integers(0, 3, (n, 1)))[..., None] % 3, 1)
    centre = np.array([distance, 0.0, 0.0])
    point = (rng.dirichlet([0.5, 0.5, 0.5], n)[..., None] * (needles + centre)).sum(1)
    target = point * (1 + rng.uniform(0.3, 1.0, (n, 1)) / distance) - centre
    corner = 1e-3 * np.array([[0.0, -1.0, -1.0], [0.0, 0.0, 1.0], [0.0, 1.0, 0.0]])  # normal along -x
    return needles, target[:, None] + corner


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("distance_au", [0.01, 0.1, 1.0])
@pytest.mark.parametrize("shadowing", [1, 2])
def test_needles_seen_edge_on(gpu_ctx, precision, distance_au, shadowing):
    from binarytpm_gb300 import lib, problem

    n = 3000
    needles, targets = _needles(n, 7, distance_au * AU_KM)
    v = np.concatenate([needles, targets]).reshape(-1, 3)
    ptr = np.concatenate([np.zeros(n + 1), np.arange(1, n + 1)]).astype(np.int32)
    prob = problem.Problem(v, np.arange(6 * n, dtype=np.int32).reshape(-1, 3), ptr, np.arange(n, dtype=np.int32),
                           np.full(n, 1e-3, np.float32), ntau=1, nx=8, polar=(distance_au, 0.0, 0.0),
                           shadowing=shadowing)
    flags = []
    for cull in "10":
        os.environ["ATPM_SHADOW_CULL"] = cull
        try:
            s = lib.Solve(gpu_ctx, prob, precision=precision)
            s.geometry_shadow()
            flags.append(s.shadow())
            s.close()
        finally:
            os.environ.pop("ATPM_SHADOW_CULL", None)
    assert np.array_equal(flags[0], flags[1]), np.count_nonzero(flags[0] != flags[1])
    assert 0 < flags[1][n:].sum() < n
