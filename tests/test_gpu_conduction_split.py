"""The lane-split depth sweep: 16, 4 or 1 lanes per facet (REFERENCE and FP64 by
the facet count, FAST by the advancing facets), every form with the same
operation sequence per node, so the results have to be equal bit for bit."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(copies, ntau, nx):
    """`copies` of one 80-facet body without view-factor lists, side by side."""
    from binarytpm_gb300 import mesh, problem

    v, f = mesh.perturbed_body(1, 0.39, 0.1, 5)
    facets = np.concatenate([f + k * len(v) for k in range(copies)])
    return problem.Problem(np.tile(v, (copies, 1)), facets.astype(np.int32), *problem.empty_lists(len(facets)),
                           ntau=ntau, nx=nx, tacc=0.05)


def _forcing(ntau):
    rng = np.random.default_rng(3)
    e = np.maximum(0.0, 1300.0 * np.sin(2 * np.pi * (np.arange(ntau) / ntau + rng.random((80, 1)))))
    return (e > 0).astype(np.int32), e.astype(np.float32)


def _run(ctx, prob, copies, precision, ti, revcap):
    from binarytpm_gb300 import lib

    s = lib.Solve(ctx, prob, precision=precision, revcap=revcap)
    lit, e = _forcing(prob.ntau)
    s.set_forcing(np.tile(lit, (copies, 1)), np.tile(e, (copies, 1)))
    s.set_thermal_inertia(ti)
    s.initialise_temperatures()
    counts = s.run()
    out = s.surface_temperature64(), s.depth_temperature(), s.converged(), counts
    s.close()
    return out


# facet counts on either side of 2, 4 warps per SM (REFERENCE) and 1/4, 2 (FP64) on 152 SMs
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ti", [0.0, 200.0])
@pytest.mark.parametrize("ntau,nx", [(48, 8), (101, 12), (53, 16), (130, 24), (245, 32)])
def test_copies_of_a_body_do_not_depend_on_the_lanes(gpu_ctx, precision, ti, ntau, nx):
    one = _run(gpu_ctx, _problem(1, ntau, nx), 1, precision, ti, 9)
    for copies in (16, 122, 250):
        many = _run(gpu_ctx, _problem(copies, ntau, nx), copies, precision, ti, 9)
        for a, b in zip(one[:3], many[:3]):
            assert np.array_equal(np.concatenate([a] * copies), b)
        assert np.array_equal(one[3] * copies, many[3])


@pytest.mark.parametrize("nx,ntau", [(8, 50), (12, 61), (16, 77), (24, 120), (32, 211), (40, 330), (48, 467), (56, 619),
                                     (64, 811)])
@pytest.mark.parametrize("freeze", [True, False])
def test_fast_forms_agree(gpu_ctx, nx, ntau, freeze):
    """16 lanes, 4 lanes and a thread per facet, on a binary with lists."""
    from binarytpm_gb300 import lib, workloads

    prob = workloads.binary_problem(gpu_ctx, 2, 1, ntau=ntau, nx=nx).with_(tacc=0.05)
    env = {"16": {"ATPM_WARP_TAIL_PER_SM": "64"}, "4": {"ATPM_WARP_TAIL_PER_SM": "1"}, "1": {"ATPM_WARP_TAIL": "0"}}
    got = {}
    for form, setting in env.items():
        old = {k: os.environ.get(k) for k in ("ATPM_WARP_TAIL", "ATPM_WARP_TAIL_PER_SM")}
        os.environ.update(setting)
        try:
            solves = [lib.Solve(gpu_ctx, prob, precision=lib.FAST, revcap=14, freeze=freeze) for _ in range(3)]
            for s, ti in zip(solves, (30.0, 200.0, 1500.0)):
                s.geometry_shadow()
                s.scattering()
                s.set_thermal_inertia(ti)
                s.initialise_temperatures()
            counts = lib.batch_run(solves)
            got[form] = [x for s, c in zip(solves, counts)
                         for x in (*s.surface_temperature(), s.depth_temperature(), s.converged(), c)]
            for s in solves:
                s.close()
        finally:
            for k, v in old.items():
                if v is None:
                    os.environ.pop(k, None)
                else:
                    os.environ[k] = v
    for form in ("16", "4"):
        for a, b in zip(got[form], got["1"]):
            assert np.array_equal(a, b), form
