"""Shadowing toward an observer close to the body: the flags of the plain drivers,
and no more triangle tests than from afar (a margin that grows with the body's size
over its distance would send whole neighbourhoods to the exact test)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shadowing", [1, 2])
@pytest.mark.parametrize("precision", [0, 2])
def test_close_observers(gpu_ctx, shadowing, precision):
    from binarytpm_gb300 import lib, workloads

    prob = workloads.binary_problem(gpu_ctx, p_subdiv=4, s_subdiv=2, ntau=45).with_(shadowing=shadowing)
    tests = []
    for au in (1.0, 1e-5, 1e-6, 3e-7, 1e-7):  # the nearest lies 15 km away, at 12 times the system's size
        s = lib.Solve(gpu_ctx, prob.with_(polar=(au, 0.1, 0.35)), precision=precision)
        s.geometry_shadow()
        got = s.shadow()
        tests.append(s.last_shadow_stats()[2])
        os.environ["ATPM_SHADOW_CULL"] = "0"
        try:
            s.geometry_shadow()
        finally:
            os.environ.pop("ATPM_SHADOW_CULL", None)
        assert np.array_equal(got, s.shadow())
        s.close()
    assert max(tests) < 1.2 * tests[0], tests
