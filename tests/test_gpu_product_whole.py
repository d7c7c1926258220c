"""FAST products whose items are dealt out by steps against the same solves in a
batch with too many items for that, bit for bit.  One group of clones of more than
half an item an SM runs its products whole; the solve alone, of fewer, in parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,ntau,entries,rows", [
    (130, 17, 20, lambda f: f % 200 < 150),              # one chunk of two 16-step groups, the last ragged
    (130, 96, 20, lambda f: True),                       # one chunk of six
    (300, 161, 40, lambda f: f % 200 < 150),             # parts that do not divide the chunk
    (700, 330, 60, lambda f: f < 130 or f >= 500),       # several chunks, a row block without a tile
    (1500, 256, 30, lambda f: f % 3 > 0),
])
def test_parts_against_whole_products(gpu_ctx, monkeypatch, nf, ntau, entries, rows):
    import torch

    from binarytpm_gb300 import lib, problem

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = -(-nf // 128)
    alone_items, clones = blocks * -(-ntau // 128), sms // (2 * blocks) + 1
    assert clones * blocks > sms // 2 and 2 * alone_items <= sms  # whole together, two parts or more alone
    monkeypatch.setenv("ATPM_TC_MIN_ENTRIES", "4")
    monkeypatch.setenv("ATPM_BATCH_STREAMS", "1")
    rng = np.random.default_rng(ntau)
    lists = [np.sort(rng.choice(nf, entries if rows(f) else 0, replace=False)) for f in range(nf)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in lists])]).astype(np.int32)
    facets = np.stack([np.arange(nf), np.arange(nf) + 1, np.arange(nf) + 2], 1).astype(np.int32)
    prob = problem.Problem(rng.normal(size=(nf + 2, 3)), facets, ptr, np.concatenate(lists).astype(np.int32),
                           rng.uniform(0.0, 0.2 / entries, ptr[-1]).astype(np.float32), ntau=ntau, nx=8)
    flux = (600.0 * rng.random((nf, ntau))).astype(np.float32)
    first = lib.Solve(gpu_ctx, prob, precision=lib.FAST, revcap=6)  # every facet, so every item, in every revolution
    first.set_forcing(np.ones((nf, ntau), np.int32), flux)
    many = [first] + [first.clone() for _ in range(clones - 1)]
    for s in many:
        s.set_thermal_inertia(40.0)
        s.initialise_temperatures()
    together = lib.batch_run(many)[0]
    want = first.surface_temperature64()
    first.set_thermal_inertia(40.0)
    first.initialise_temperatures()
    assert np.array_equal(together, first.run())
    assert np.array_equal(first.surface_temperature64(), want)
    for s in many:
        s.close()
