"""Gauss-Seidel scattering in level order (k_multi_levels) against the
facet-by-facet restatement, bit for bit: every steps-per-CTA form (8, 4, 2 or 1
lanes a facet by the facet count), remainders of the steps, rows of every kind
(empty, only lower, only higher neighbours), and unsorted lists, which keep the
facet-by-facet kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(nf, ntau, seed, ascending=True):
    from binarytpm_gb300 import problem

    rng = np.random.default_rng(seed)
    rows = []
    for f in range(nf):
        n = int(rng.integers(0, 7)) if f % 5 else 0
        near = np.clip(f + rng.integers(-40, 41, n), 0, nf - 1)
        row = np.unique(np.concatenate([near, rng.integers(0, nf, n // 3)]))
        row = row[row != f]
        rows.append(row if ascending else rng.permutation(row))
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    idx = np.concatenate(rows).astype(np.int32)
    v = rng.normal(size=(nf + 2, 3))
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    return problem.Problem(v, facets, ptr, idx, rng.uniform(0.0, 0.12, len(idx)).astype(np.float32), ntau=ntau, nx=8,
                           shadowing=0, albedo=0.3, scattering_accuracy=1e-4)


def _restated(prob, cos, lit, solar, real):
    """Single scattering, then Gauss-Seidel sweeps in facet order, all steps as
    numpy vectors, each step stopping at its own convergence."""
    r = real
    solar, alb, acc = r(solar), r(prob.albedo), r(prob.scattering_accuracy)
    vf = prob.dep_vf.astype(real)
    sp = (solar * cos) * lit
    e = sp.copy()
    lists = [range(prob.dep_ptr[f], prob.dep_ptr[f + 1]) for f in range(prob.nf)]
    for f, ks in enumerate(lists):
        for k in ks:
            g = prob.dep_idx[k]
            e[f] = e[f] + (((vf[k] * solar) * alb) * cos[g]) * lit[g]
    po = alb * e
    pn = po.copy()
    active = np.ones(prob.ntau, bool)
    while active.any():
        for f, ks in enumerate(lists):
            if not len(ks):
                continue
            after, before = np.zeros(prob.ntau, real), np.zeros(prob.ntau, real)
            for k in ks:
                g = prob.dep_idx[k]
                if g > f:
                    after = after + vf[k] * po[g]
                else:
                    before = before + vf[k] * pn[g]
            pn[f] = np.where(active, alb * ((sp[f] + after) + before), pn[f])
        active &= (np.abs(pn - po) > acc).any(0)
        po = pn.copy()
    return pn / alb


@pytest.mark.parametrize("nf,ntau", [(1, 1), (37, 2), (300, 9), (7041, 8), (7040, 13), (14081, 7), (28161, 5),
                                     (56321, 3)])
@pytest.mark.parametrize("precision", ["reference", "fp64"])
def test_level_order_is_facet_order(gpu_ctx, nf, ntau, precision):
    _check(gpu_ctx, _problem(nf, ntau, nf), precision)


def test_unsorted_lists(gpu_ctx):
    _check(gpu_ctx, _problem(301, 10, 4, ascending=False), "reference")


def _check(ctx, prob, precision):
    from binarytpm_gb300 import lib

    s = lib.Solve(ctx, prob, precision=lib.PRECISIONS[precision])
    s.geometry_shadow()
    s.scattering()
    again = s.clone()
    again.scattering()
    real = np.float32 if precision == "reference" else np.float64
    got = s.illumination()
    assert np.array_equal(got, again.illumination())
    want = _restated(prob, s.cosillum().astype(real), s.shadow().astype(real), s.solar(), real)
    if precision == "reference":
        assert np.array_equal(got, want.astype(np.float32))
    else:  # cosillum is read back in 32 bits (2^-24 a term, all terms positive), and a step whose last change lies
        # beside the accuracy may take one sweep more or less
        assert np.all(np.abs(got - want) <= 2.0 ** -22 * np.abs(want) + 2 * prob.scattering_accuracy / prob.albedo)
    s.close()
    again.close()
