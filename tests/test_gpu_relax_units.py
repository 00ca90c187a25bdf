"""Relaxation where the storage type's range matters: boxes whose units make a normalised
field very large or very small, so that merged steps between renormalisations have little
of the range left, and a potential with an infinite wall (no merging), against the FP64
oracle, which renormalises after every step (complex128 1e-12, complex64 1e-5)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def run(ses, oracle, prec, g, V, dtau, psi, steps, mass=1.0):
    want = oracle.relax3d(g.box, g.dims, V, dtau, psi, steps, mass=mass)
    op = ses.ImaginaryTimePropagator3D(g, V, dtau, mass=mass, precision=prec, psi0=psi)
    e = op.relax_resident(steps)
    got = op.readback()
    op.close()
    assert np.all(np.isfinite(got.view(np.float64))) and np.isfinite(e)
    return rel(got, want)


# box lengths of 12 units; a unit squared per mass and step of imaginary time stays 0.02
@pytest.mark.parametrize("prec,tol,unit", [("c64", 1e-5, 1e-12), ("c64", 1e-5, 1e-6), ("c64", 1e-5, 1e10),
                                           ("c64", 1e-5, 1e13), ("c128", 1e-12, 1e-60), ("c128", 1e-12, 1e60)])
@pytest.mark.parametrize("scale", [2.0, -2.0])
def test_units_far_from_one(ses, oracle, prec, tol, unit, scale):
    n = 20
    dtau = 0.02 * unit * unit
    g = ses.Grid3D(*(ses.Grid1D(-6.0 * unit, 6.0 * unit, n) for _ in range(3)))
    x = np.asarray(g.x.coords()) / unit
    r2 = (x ** 2)[None, None, :] + (x ** 2)[None, :, None] + (x ** 2)[:, None, None]
    V = (scale / 0.02 + 0.5 * r2).reshape(-1) / (unit * unit)  # e^-+2 a step over the whole box
    psi = np.exp(-r2 / 4.0).reshape(-1).astype(complex)
    psi /= np.sqrt(np.sum(np.abs(psi) ** 2)) * g.cell_volume() ** 0.5
    assert run(ses, oracle, prec, g, V, dtau, psi, 40) <= tol


@pytest.mark.parametrize("prec,tol", [("c128", 1e-12), ("c64", 1e-5)])
@pytest.mark.parametrize("wall", [np.inf, 1e300])
def test_infinite_wall(ses, oracle, prec, tol, wall):
    g = ses.Grid3D(*(ses.Grid1D(-6.0, 6.0, 20) for _ in range(3)))
    x = np.asarray(g.x.coords())
    r2 = (x ** 2)[None, None, :] + (x ** 2)[None, :, None] + (x ** 2)[:, None, None]
    V = np.where(r2 > 25.0, wall, 0.5 * r2).reshape(-1)
    psi = np.exp(-r2 / 4.0).reshape(-1).astype(complex)
    assert run(ses, oracle, prec, g, V, 0.02, psi, 37) <= tol
