"""The autotuner keeps its choices apart for batches whose revolutions run a
thread per facet and for smaller ones, which share a facet's column between lanes
and have no conduction variant to choose."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(ctx, nf):
    from binarytpm_gb300 import lib, problem

    ntau = 16
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    prob = problem.Problem(np.random.default_rng(0).normal(size=(nf + 2, 3)), facets, *problem.empty_lists(nf), ntau=ntau,
                           nx=8)
    s = lib.Solve(ctx, prob, precision=lib.FAST, revcap=6)
    s.set_forcing(np.ones((nf, ntau), np.int32), np.full((nf, ntau), 300.0, np.float32))
    s.set_thermal_inertia(100.0)
    s.initialise_temperatures()
    s.run()
    out = s.last_run_config()
    s.close()
    return out


def test_small_batches_do_not_choose_for_larger_ones(gpu_ctx, monkeypatch):
    import torch

    from binarytpm_gb300 import lib

    line = 56 * torch.cuda.get_device_properties(0).multi_processor_count
    small, large = line - 64, line + 64
    # one power-of-two class of facet blocks
    assert (-(-small // 128) - 1).bit_length() == (-(-large // 128) - 1).bit_length()
    ctx = lib.Context(0)  # nothing tuned yet
    assert _run(ctx, small)[::2] == (4, True)
    assert _run(ctx, large)[2]
    assert not _run(ctx, small)[2] and not _run(ctx, large)[2]
    ctx.close()
    # without the lane-split sweep a small batch is of the larger ones' kind
    ctx = lib.Context(0)
    assert _run(ctx, large)[2]
    monkeypatch.setenv("ATPM_WARP_TAIL", "0")
    assert not _run(ctx, small)[2]
    ctx.close()


def test_dealt_out_products_keep_the_default_depth(gpu_ctx):
    """A few row blocks' items are dealt out in parts at a ring depth of their own."""
    from binarytpm_gb300 import lib, problem

    nf, ntau = 256, 256
    rng = np.random.default_rng(1)
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    idx = np.sort(np.stack([rng.choice(nf, 40, replace=False) for _ in range(nf)]), axis=1).reshape(-1)
    prob = problem.Problem(rng.normal(size=(nf + 2, 3)), facets, (40 * np.arange(nf + 1)).astype(np.int32),
                           idx.astype(np.int32), np.full(40 * nf, 1e-3, np.float32), ntau=ntau, nx=8)
    depths = set()
    for _ in range(8):
        ctx = lib.Context(0)
        s = lib.Solve(ctx, prob, precision=lib.FAST, revcap=6)
        s.set_forcing(np.ones((nf, ntau), np.int32), np.full((nf, ntau), 300.0, np.float32))
        s.set_thermal_inertia(100.0)
        s.initialise_temperatures()
        s.run()
        depths.add(s.last_run_config()[::2] + (s.last_run_config()[1],))
        s.close()
        ctx.close()
    assert len(depths) == 1 and depths.pop()[:2] == (4, True)
