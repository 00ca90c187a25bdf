"""Run-time-plan passes (lengths without a compiled plan, dipole-driven steps, runs
of a 1D line in one launch) against the FP64 oracle: lengths of one, two, three and
more stages, every radix, line counts that do not fill a tile, and both passes'
reversed order.

Tolerances are those of the step anywhere in this suite: complex128 1e-12 relative L2
a step, complex64 1e-5 over a run, transforms 1e-14 / 5e-7 times log2 N."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


# 1D: one stage (2 .. 15), two (18 .. 250), three (500, 1080, 1024, 2048, 4096), four and five (2187, 3125)
LINES = [2, 3, 5, 9, 15, 18, 25, 27, 36, 50, 81, 90, 100, 120, 135, 144, 180, 200, 225, 240, 250, 256, 500, 625, 1024,
         1080, 2048, 2187, 3125, 3750, 4096]


@pytest.mark.parametrize("n", LINES)
def test_lines_transform_and_step(ses, oracle, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    for inverse in (False, True):
        want = oracle.fft3d(a, (n, 1, 1), inverse=inverse)
        f = ses.ifft if inverse else ses.fft
        assert rel(f(a), want) < 1e-14 * max(1.0, math.log2(n))
        assert rel(f(a, precision="c64"), want) < 5e-7 * max(1.0, math.log2(n))
    g = ses.line_grid(ses.Grid1D(-6.0, 6.0, n))
    V = 0.5 * np.asarray(g.x.coords()) ** 2
    psi = oracle.gaussian3d(g.box, g.dims, (0.5, 0.0, 0.0), (1.0, 1.0, 1.0), (0.3, 0.0, 0.0))
    mask = 1.0 - 0.1 * rng.random(n)  # one axis: any mask is separable
    for prec in ("c128", "c64"):
        op = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
        op.set_absorber(mask)
        for steps in (1, 2, 7):
            op.upload_state(psi)
            op.advance(steps, absorb=True)
            want = oracle.step3d(g.box, g.dims, V, 0.01, psi, steps, mask=mask)
            assert rel(op.readback(), want) < (steps * 1e-12 if prec == "c128" else 1e-5), (prec, steps)
        op.close()


@pytest.mark.parametrize("prec", ["c128", "c64"])
def test_line_runs_split_anywhere_give_the_same_bits(ses, oracle, prec):
    n = 360
    g = ses.line_grid(ses.Grid1D(-8.0, 8.0, n))
    V = 0.5 * np.asarray(g.x.coords()) ** 2
    psi = oracle.gaussian3d(g.box, g.dims, (0.5, 0.0, 0.0), (1.0, 1.0, 1.0), (0.3, 0.0, 0.0))
    outs = []
    for parts in ((1100,), (1024, 76), (1, 2, 97, 1000)):  # the launch limit is inside the first
        op = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
        op.set_absorber(np.linspace(0.999, 1.0, n))
        for k in parts:
            op.advance(k, absorb=True)
        outs.append(op.readback())
        op.close()
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])


BOXES = [(5, 3, 2), (9, 25, 15), (18, 27, 20), (30, 45, 50), (120, 10, 9), (10, 120, 9), (9, 10, 120), (225, 4, 6),
         (6, 240, 5), (4, 6, 250), (75, 64, 36), (100, 90, 1), (81, 1, 40), (1, 50, 45), (1, 1, 54), (48, 500, 1),
         (2000, 4, 1), (4, 2048, 1), (3, 3125, 1)]


@pytest.mark.parametrize("dims", BOXES, ids=["x".join(map(str, d)) for d in BOXES])
def test_boxes_step_and_observe(ses, oracle, dims):
    box = tuple(v for d in dims for v in ((-6.0, 6.0) if d > 1 else (0.0, 1.0)))
    live = [1.0 if d > 1 else 0.0 for d in dims]
    V = oracle.harmonic3d(box, dims, 0.7, tuple(0.2 * a for a in live))
    psi = oracle.gaussian3d(box, dims, tuple(0.5 * a for a in live), (1.4, 1.3, 1.2), tuple(0.3 * a for a in live))
    mask = oracle.mask3d(box, dims, 1.5, 1)
    g = ses.Grid3D(*(ses.Grid1D(box[2 * a], box[2 * a + 1], dims[a]) for a in range(3)))
    for prec in ("c128", "c64"):
        op = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
        op.set_absorber(mask)
        op.advance(10, absorb=True)
        want = oracle.step3d(box, dims, V, 0.01, psi, 10, mask=mask)
        got = op.readback()
        assert rel(got, want) < (1e-11 if prec == "c128" else 1e-5), prec
        # <T> of the field read back, by numpy (relative error of an FP32 transform's energy: 1e-5)
        k = [2 * math.pi * np.fft.fftfreq(a.n, a.spacing()) if a.n > 1 else np.zeros(1) for a in (g.x, g.y, g.z)]
        phi = np.abs(np.fft.fftn(got.reshape(g.shape))) ** 2
        k2 = k[0][None, None, :] ** 2 + k[1][None, :, None] ** 2 + k[2][:, None, None] ** 2
        t = float((0.5 * k2 * phi).sum() / phi.sum())
        assert abs(op.observe()["energy_t"] - t) <= (1e-10 if prec == "c128" else 1e-5) * max(t, 1e-3)
        op.close()


@pytest.mark.parametrize("prec", ["c128", "c64"])
@pytest.mark.parametrize("dims", [(36, 20, 15), (64, 32, 5), (160, 9, 1), (27, 256, 1), (16, 1, 30),
                                  (4096, 3, 1)])
def test_driven_steps_on_run_time_plans(ses, oracle, dims, prec):
    box = tuple(v for d in dims for v in ((-8.0, 8.0) if d > 1 else (0.0, 1.0)))
    live = [1.0 if d > 1 else 0.0 for d in dims]
    V = oracle.harmonic3d(box, dims, 0.8)
    psi = oracle.gaussian3d(box, dims, (1.0, -0.5 * live[1], 0.0), (1.2, 1.2, 1.2), (0.4, 0.0, 0.0))
    g = ses.Grid3D(*(ses.Grid1D(box[2 * a], box[2 * a + 1], dims[a]) for a in range(3)))
    op = ses.SplitOperator3D(g, V, 0.02, precision=prec, psi0=psi)
    op.advance_driven(12, (0.6, 0.8, 0.3), 0.5, 1.3, 0.1)
    want = oracle.driven_step3d(box, dims, V, 0.02, psi, 12, (0.6, 0.8, 0.3), 0.5, 1.3, 0.1)
    assert rel(op.readback(), want) <= (1.2e-11 if prec == "c128" else 1e-5)
    op.close()
