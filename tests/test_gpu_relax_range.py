"""Relaxation in merged runs between renormalisations: potentials whose steps scale
the field so much that runs get short (down to one step) or that grow it, a field
that comes in far from normalised, and the energy of the last renormalisation for
run lengths around the merge limit -- against the FP64 oracle, which renormalises
after every step (complex128 1e-12, complex64 1e-5, as the plain relaxation)."""

import math

import numpy as np
import pytest

from shoeridingerequationsolver_b200 import scenes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


# exp(-offset dtau) a step: 1 .. e^-40, e^40 (complex64 keeps weights as w - 1, which
# resolves no weight below 1e-7: e^-4 is its steepest here)
@pytest.mark.parametrize("prec,tol,offset", [("c128", 1e-12, v) for v in (0.0, 40.0, 2000.0, -2000.0)]
                         + [("c64", 1e-5, v) for v in (0.0, 40.0, 200.0, -2000.0)])
@pytest.mark.parametrize("nsteps", [1, 2, 35, 71])
def test_relax_with_steep_potentials(ses, oracle, prec, tol, offset, nsteps):
    g = scenes.cube_grid(-6.0, 6.0, 20)
    dtau = 0.02
    V = scenes.harmonic(g, 1.0, (0.2, 0.0, -0.1)) + offset
    psi = scenes.gaussian(g, (0.8, -0.4, 0.3), (1.2, 0.9, 1.1), (0.0, 0.0, 0.0))
    want = oracle.relax3d(g.box, g.dims, V, dtau, psi, nsteps)
    op = ses.ImaginaryTimePropagator3D(g, V, dtau, precision=prec, psi0=1e3 * psi)
    e = op.relax_resident(nsteps)
    got = op.readback()
    assert rel(got, want) <= tol
    if nsteps > 1:  # the last step's energy: that of one more oracle step from the field before it
        before = oracle.relax3d(g.box, g.dims, V, dtau, psi, nsteps - 1)
        hv = np.exp(-0.5 * V * dtau)
        k = 2 * math.pi * np.fft.fftfreq(20, 12.0 / 20)
        k2 = (k ** 2)[None, None, :] + (k ** 2)[None, :, None] + (k ** 2)[:, None, None]
        f = np.fft.ifftn(np.exp(-0.5 * k2 * dtau) * np.fft.fftn((hv * before).reshape(g.shape))).reshape(-1) * hv
        n2 = float(np.sum(np.abs(f) ** 2) * g.cell_volume())
        assert abs(e + math.log(n2) / (2 * dtau)) <= (1e-9 if prec == "c128" else 1e-3) * max(1.0, abs(offset))
    op.close()


@pytest.mark.parametrize("prec,tol", [("c128", 1e-12), ("c64", 1e-5)])
@pytest.mark.parametrize("dims", [(360, 1, 1), (50, 36, 1), (64, 64, 1), (30, 1, 24)])
def test_relax_on_lines_and_planes(ses, oracle, prec, tol, dims):
    box = tuple(v for d in dims for v in ((-6.0, 6.0) if d > 1 else (0.0, 1.0)))
    live = [1.0 if d > 1 else 0.0 for d in dims]
    V = oracle.harmonic3d(box, dims, 1.0, tuple(0.2 * a for a in live))
    psi = oracle.gaussian3d(box, dims, tuple(0.6 * a for a in live), (1.2, 0.9, 1.1), (0.0, 0.0, 0.0))
    g = ses.Grid3D(*(ses.Grid1D(box[2 * a], box[2 * a + 1], dims[a]) for a in range(3)))
    want = oracle.relax3d(box, dims, V, 0.01, psi, 40)
    for every in (1, 7):
        op = ses.ImaginaryTimePropagator3D(g, V, 0.01, precision=prec, psi0=psi)
        op.relax_resident(40, renorm_every=every)
        assert rel(op.readback(), want) <= tol, every
        op.close()
