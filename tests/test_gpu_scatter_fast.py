"""FAST scattering rounds as it always has, bit for bit: single scattering adds each
rounded term in list order, a Jacobi sweep sums every other entry with fused
multiply-adds and adds the rounded sunlight.  One ulp of the forcing is enough to move
the revolution in which a facet counts as converged."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _fma(a, b, c):
    """a b + c rounded once to 32 bits."""
    exact = Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c))
    f = F(float(exact))
    near = [f, np.nextafter(f, F(-np.inf)), np.nextafter(f, F(np.inf))]
    return min(near, key=lambda x: (abs(Fraction(float(x)) - exact), int(x.view(np.uint32)) & 1))


def _restated(prob, cos, lit, solar, multiple):
    solar, alb, acc = F(solar), F(prob.albedo), F(prob.scattering_accuracy)
    lists = [list(zip(prob.dep_idx[a:b], prob.dep_vf[a:b])) for a, b in zip(prob.dep_ptr, prob.dep_ptr[1:])]
    direct = (solar * cos) * lit
    e = direct.copy()
    for f, entries in enumerate(lists):
        for g, v in entries:
            e[f] = e[f] + (((v * solar) * alb) * cos[g]) * lit[g]
    if not multiple:
        return e
    old = alb * e
    while True:
        new = np.empty_like(old)
        for f, entries in enumerate(lists):
            for s in range(prob.ntau):
                part = [F(0), F(0)]
                for k, (g, v) in enumerate(entries):
                    part[k & 1] = _fma(v, old[g, s], part[k & 1])
                new[f, s] = alb * (direct[f, s] + (part[0] + part[1]))
        done = not (np.abs(new - old) > acc).any()
        old = new
        if done:
            return old / alb


@pytest.mark.parametrize("nf,ntau,multiple", [(40, 9, 0), (300, 33, 0), (40, 9, 1), (131, 6, 1)])
def test_fast_scattering_bits(gpu_ctx, nf, ntau, multiple):
    from binarytpm_gb300 import lib, problem

    rng = np.random.default_rng(nf)
    rows = [np.unique(rng.integers(0, nf, rng.integers(0, 12))) for _ in range(nf)]
    rows = [r[r != f] for f, r in enumerate(rows)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    prob = problem.Problem(rng.normal(size=(nf + 2, 3)), facets, ptr, np.concatenate(rows).astype(np.int32),
                           rng.uniform(0.0, 0.1, ptr[-1]).astype(np.float32), ntau=ntau, nx=8, shadowing=0, albedo=0.3,
                           multiple_scattering=multiple)
    s = lib.Solve(gpu_ctx, prob, precision=lib.FAST)
    s.geometry_shadow()
    s.scattering()
    want = _restated(prob, s.cosillum(), s.shadow().astype(np.float32), s.solar(), multiple)
    assert np.array_equal(s.illumination(), want)
    s.close()
