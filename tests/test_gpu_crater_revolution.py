"""Crater revolutions: steps in batches of eight and, beyond the resident CTAs,
in segments.  REFERENCE is held to a restatement of the module's float
expressions bit for bit at sub-facet and step counts around the batch and the
view-factor loop's unrolling; craters of more facets than fit the GPU at once
are held to the same facets in craters that do."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS, SIGMA, TACC = np.float32(0.9), np.float32(5.67e-8), np.float32(0.005)


def _inputs(nf, ntau, nsf, seed):
    rng = np.random.default_rng(seed)
    e = rng.uniform(0.0, 1300.0, (nf, ntau, nsf)).astype(np.float32)
    return {"V": rng.uniform(0.0, 0.8 / nsf, (nsf, nsf)).astype(np.float32), "RI": e,
            "RGH": rng.uniform(0.0, 30.0, e.shape).astype(np.float32),
            "ti": rng.uniform(20.0, 900.0, nf).astype(np.float32),
            "alb": rng.uniform(0.0, 0.3, nf).astype(np.float32),
            "start": rng.uniform(150.0, 350.0, e.shape).astype(np.float32)}


def _run(ctx, x, nx, precision, revs, rows=slice(None)):
    from binarytpm_gb300 import lib

    ri = x["RI"][rows]
    nf, ntau, nsf = ri.shape
    c = lib.Crater(ctx, nf, ntau, nx, nsf, precision)
    fac = np.stack([np.arange(nsf) % 60, (np.arange(nsf) + 1) % 60, (np.arange(nsf) + 2) % 60], 1)
    c.set_model(np.random.default_rng(0).normal(size=(60, 3)), fac, np.zeros((nsf, 2, 3)), x["V"], 2.26 * 3600.0)
    c.set_properties(np.zeros(nf, np.uint8), x["alb"][rows], x["ti"][rows])
    c.set_array(c.ILLUMINATION, ri)
    c.set_array(c.GLOBAL_HEATING, x["RGH"][rows])
    c.initialise_temperatures(float(EPS), float(SIGMA))
    c.set_temperatures(x["start"][rows])
    first = c.temperatures()[2]
    for _ in range(revs):
        c.inertia_difference(float(EPS), float(SIGMA), float(TACC))
    out = c.temperatures()
    c.close()
    return first, out


def _restated(x, nx, column, revs):
    """GPU_code.cu:377-490 in float, operand by operand ([nf][nx + 1][nsf] columns)."""
    from oracle import oracle

    f = np.float32
    nf, ntau, nsf = x["RI"].shape
    pi = f(4.0) * np.arctan(f(1.0))
    es = f(EPS * SIGMA)
    es4 = f(4.0) * es
    dz = f(8.0) / f(nx)
    m0 = ((f(2.0) * pi) / f(ntau)) / (dz * dz)
    m1 = ((x["ti"] * np.sqrt((f(2.0) * pi) / f(2.26 * 3600.0))) / dz)[:, None]
    oma = (f(1.0) - x["alb"])[:, None]
    T, s1 = column.copy(), x["start"].copy()
    s0 = np.zeros_like(s1)
    for _ in range(revs):
        for s in range(ntau):
            old = s1[:, s].copy()
            t0 = T[:, 0].copy()
            for i in range(1, nx):
                t1 = T[:, i].copy()
                T[:, i] = t1 + m0 * ((T[:, i + 1] - f(2.0) * t1) + t0)
                t0 = t1
            T[:, nx] = T[:, nx - 1]
            s0[:, s] = old
            w = es * oracle.glibc_powf(old.ravel(), 4.0).reshape(old.shape)
            inc = x["RGH"][:, s].copy()
            for i in range(nsf):
                inc = inc + w[:, i:i + 1] * x["V"][i][None, :]
            m2 = oma * x["RI"][:, s] + inc
            tr, dt = T[:, 0].copy(), np.ones_like(old)
            while (go := dt >= TACC / f(10.0)).any():
                t3 = ((es * tr) * tr) * tr
                new = tr + ((m2 + m1 * (T[:, 1] - tr)) - t3 * tr) / (m1 + ((es4 * tr) * tr) * tr)
                dt = np.where(go, np.abs(new - tr), dt)
                tr = np.where(go, new, tr)
            T[:, 0] = tr
            s1[:, s] = tr
    return s0, s1, T


@pytest.mark.parametrize("nsf,ntau,nx", [(5, 30, 8), (37, 31, 8), (100, 33, 8), (128, 41, 8), (99, 72, 12)])
def test_reference_is_the_modules_order(gpu_ctx, nsf, ntau, nx):
    from binarytpm_gb300 import lib

    x = _inputs(3, ntau, nsf, nsf)
    first, got = _run(gpu_ctx, x, nx, lib.REFERENCE, 2)
    for a, b in zip(got, _restated(x, nx, first, 2)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("precision", ["REFERENCE", "FAST"])
@pytest.mark.parametrize("ntau", [30, 64, 97])
def test_segments_do_not_change_a_facet(gpu_ctx, precision, ntau):
    from binarytpm_gb300 import lib

    x = _inputs(1400, ntau, 20, ntau)
    prec = getattr(lib, precision)
    _, whole = _run(gpu_ctx, x, 8, prec, 3)
    for rows in (slice(0, 200), slice(700, 1100), slice(1200, 1400)):
        _, part = _run(gpu_ctx, x, 8, prec, 3, rows)
        for a, b in zip(whole, part):
            assert np.array_equal(a[rows].view(np.uint32), b.view(np.uint32))
