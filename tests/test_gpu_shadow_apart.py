"""All-pairs visibility of small bodies far apart: the flags of the plain driver, in a
time that does not follow the empty space between the bodies."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_bodies_far_apart(gpu_ctx):
    from binarytpm_gb300 import lib, mesh, problem

    took = []
    for separation in (1.2, 10.0, 60.0, 500.0):
        v, f = mesh.binary_system(mesh.perturbed_body(3, 0.39, 0.05, 1), mesh.perturbed_body(3, 0.08, 0.08, 2), separation)
        prob = problem.Problem(v, f.astype(np.int32), *problem.empty_lists(len(f)), ntau=200, nx=8, polar=(1.2, 0.0, 0.35),
                               shadowing=2)
        s = lib.Solve(gpu_ctx, prob, precision=lib.REFERENCE)
        times = []
        for _ in range(3):
            s.geometry_shadow()
            times.append(s.last_shadow_stats()[0])
        took.append(min(times))
        got = s.shadow()
        os.environ["ATPM_SHADOW_CULL"] = "0"
        try:
            s.geometry_shadow()
        finally:
            os.environ.pop("ATPM_SHADOW_CULL", None)
        assert np.array_equal(got, s.shadow())
        s.close()
    assert max(took) < 20 * took[0], took
