"""The crater's partial shadows and scattering against restatements of the
module's float expressions (GPU_code.cu:152-304), bit for bit in REFERENCE:
directions and steps in groups of four, Suns overhead, grazing, along an axis and
of any length, shapes from the crater's own size to a hundred times it, fractions
other than 0 and 1, and step counts around the groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


def _multipliers():
    m = np.zeros((100, 2), F)
    for k in range(1, 11):
        for l in range(1, k + 1):
            m[(k - 1) ** 2 + 2 * (l - 1)] = F(k) - F(1) / F(3), F(l) - F(2) / F(3)
    for k in range(2, 11):
        for l in range(1, k):
            m[(k - 1) ** 2 + 2 * (l - 1) + 1] = F(k) - F(2) / F(3), F(l) - F(1) / F(3)
    return m


def _crater(ctx, nf, ntau, nsf, precision, size=1.0):
    """Triangles on a bowl of radius 10 x size (the rim's radius is 10)."""
    from binarytpm_gb300 import lib

    rng = np.random.default_rng(nsf)
    r, phi = 10.0 * np.sqrt(rng.random(60)), 2 * np.pi * rng.random(60)
    v = (size * np.stack([r * np.cos(phi), r * np.sin(phi), 0.05 * r * r - 5.0], 1)).astype(F)
    fac = np.stack([np.arange(nsf) % 60, (np.arange(nsf) + 7) % 60, (np.arange(nsf) + 13) % 60], 1).astype(np.int32)
    a, b, e = (v[fac[:, k]] for k in range(3))
    tri = np.stack([F(-1) * (e - a) / F(10), (b - a) / F(10)], 1)
    vf = rng.uniform(0.0, 0.8 / nsf, (nsf, nsf)).astype(F)
    c = lib.Crater(ctx, nf, ntau, 16, nsf, lib.PRECISIONS[precision])
    c.set_model(v, fac, tri, vf, 2.26 * 3600.0)
    return c, v, fac, tri, vf, rng


def _suns(rng, n):
    s = rng.normal(size=(n, 3)) * np.exp(rng.normal(size=(n, 1)))
    s[:, 2] = np.abs(s[:, 2]) * np.exp(-3.0 * rng.random(n))
    for k, special in enumerate([(0, 0, 1), (1, 0, 0), (1, 0, 1e-20), (0, -1, 0.5), (1e-3, 0, 1), (3, 4, 0.0)]):
        if k < n:
            s[k] = special
    return s.astype(F)


def _shadow(v, fac, tri, suns, flags, start):
    """sfcpartialshadow for every (direction, sub-facet)."""
    out = start.copy()
    at = v[fac[:, 2]]
    with np.errstate(all="ignore"):
        n = np.sqrt(suns[:, 0] * suns[:, 0] + suns[:, 1] * suns[:, 1])
        w = suns / n[:, None]
        slope = np.abs(w[:, 2]) / np.sqrt(w[:, 0] * w[:, 0] + w[:, 1] * w[:, 1])
        w0, w1, slope = w[:, :1], w[:, 1:2], slope[:, None]
        for m0, m1 in _multipliers():
            mp = ((at + m0 * tri[:, 0]) + m1 * tri[:, 1])[None]
            t = (F(-1) * w1) * mp[..., 0] + w0 * mp[..., 1]
            rad = np.sqrt(F(100) - t * t)
            u = (w0 * mp[..., 0] + w1 * mp[..., 1]) - rad
            hit = (mp[..., 2] <= slope * u) & (out != 0) & flags[:, None]
            out = np.where(hit, out - F(1) / F(100), out)
            out = np.where(flags[:, None] & (out < 0), F(0), out)
    return out


@pytest.mark.parametrize("nf,ntau,nsf", [(1, 1, 100), (3, 7, 100), (20, 33, 100), (5, 40, 37), (2, 6, 128)])
@pytest.mark.parametrize("size", [0.98, 1.3, 100.0])
def test_partial_shadow(gpu_ctx, nf, ntau, nsf, size):
    c, v, fac, tri, _, rng = _crater(gpu_ctx, nf, ntau, nsf, "reference", size)
    suns = _suns(rng, nf * ntau)
    flags = rng.random(nf * ntau) < 0.8
    start = rng.choice([0.0, 1.0, 1.0, 1.0, 0.5, 0.015], (nf * ntau, nsf)).astype(F)
    c.set_array(c.SUN_VECTOR, suns)
    c.set_array(c.SHADOW, flags.astype(np.int32))
    c.set_array(c.SFC_SHADOW, start)
    c.partial_shadow()
    got = c.get_array(c.SFC_SHADOW).reshape(start.shape)
    c.close()
    assert np.array_equal(got, _shadow(v, fac, tri, suns, flags, start))


@pytest.mark.parametrize("nf,ntau,nsf", [(1, 1, 100), (3, 7, 100), (9, 12, 37), (2, 6, 128)])
@pytest.mark.parametrize("multiple", [False, True])
def test_scattering(gpu_ctx, nf, ntau, nsf, multiple):
    c, _, _, _, vf, rng = _crater(gpu_ctx, nf, ntau, nsf, "reference")
    shape = (nf, ntau, nsf)
    lit, angle = rng.random(shape).astype(F), rng.random(shape).astype(F)
    lit[:, ::3] = 0.0  # dark steps converge at once
    more = (30.0 * rng.random(shape)).astype(F)
    alb = rng.uniform(0.02, 0.5, nf).astype(F)
    c.set_properties(np.zeros(nf, np.uint8), alb, np.full(nf, 200.0))
    c.set_array(c.SFC_SHADOW, lit)
    c.set_array(c.SFC_SUN_ANGLE, angle)
    c.set_array(c.GLOBAL_ILLUMINATION, more)
    c.scattering(1361.0, 1e-3, multiple)
    got = c.get_array(c.ILLUMINATION)
    c.close()
    solar, alb = F(1361.0), alb[:, None, None]
    ill = solar * lit * angle + more
    power = solar * angle * lit + more
    tot = ill.copy()
    for i in range(nsf):
        tot = tot + (vf[i] * alb) * ill[..., i:i + 1]
    tot = np.where(tot <= 0, F(0), tot)
    if multiple:
        old, going = alb * tot, np.ones((nf, ntau, 1), bool)
        while going.any():
            total = np.zeros(shape, F)
            for i in range(nsf):
                total = total + vf[i] * old[..., i:i + 1]
            new = np.where(going, alb * (power + total), old)
            going &= (np.abs(new - old) > F(1e-3)).any(-1, keepdims=True)
            old = new
        tot = old / alb
    assert np.array_equal(got, tot)
