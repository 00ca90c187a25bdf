"""Observables and norm / peak on fields whose point count sits at the edges of the
reductions: fewer points than a thread block, one trip of the grid and one more
point, odd axis lengths, more partial rows than one CTA folds in a trip.

The sums are FP64 over at most N = 3e6 terms in a tree of partial sums, so each is
within N eps of the sum numpy forms (the readings here are within 1e-11 for terms
of one sign; positions and momenta are compared on the scale of the box and of the
largest wavenumber)."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(1, 1, 1), (5, 3, 1), (27, 25, 3), (64, 16, 1), (64, 4, 4), (25, 40, 1), (45, 81, 1), (125, 75, 27),
        (128, 128, 128), (2048, 1, 1), (8192, 1, 1), (160, 135, 128)]


def expected(g, V, psi, xlo, xhi):
    x, y, z = (a.coords() for a in (g.x, g.y, g.z))
    f = psi.reshape(g.shape)
    w = np.abs(f) ** 2
    k = [np.zeros(1) if a.n == 1 else 2 * math.pi * np.fft.fftfreq(a.n, a.spacing()) for a in (g.x, g.y, g.z)]
    phi = np.abs(np.fft.fftn(f)) ** 2
    along = [w.sum((0, 1)), w.sum((0, 2)), w.sum((1, 2))]
    kal = [phi.sum((0, 1)), phi.sum((0, 2)), phi.sum((1, 2))]
    r = (x, y, z)
    mean = [float(r[a] @ along[a] / w.sum()) for a in range(3)]
    return dict(norm=w.sum() * g.cell_volume(), energy_v=float((V.reshape(g.shape) * w).sum() / w.sum()),
                energy_t=float(sum((0.5 * k[a] ** 2) @ kal[a] for a in range(3)) / phi.sum()),
                p_range=float(along[0][(x >= xlo) & (x < xhi)].sum() * g.cell_volume()), mean_pos=mean,
                sigma_pos=[math.sqrt(max(0.0, float((r[a] - mean[a]) ** 2 @ along[a] / w.sum()))) for a in range(3)],
                mean_mom=[float(k[a] @ kal[a] / phi.sum()) for a in range(3)], peak=float(w.max()))


@pytest.mark.parametrize("prec", ["c128", "c64"])
@pytest.mark.parametrize("dims", DIMS, ids=["x".join(map(str, d)) for d in DIMS])
def test_observables_at_reduction_edges(ses, dims, prec):
    rng = np.random.default_rng(sum(dims))
    g = ses.Grid3D(*(ses.Grid1D(-4.0, 5.0, n) if n > 1 else ses.Grid1D(0.0, 1.0, 1) for n in dims))
    N = g.size()
    psi = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    if prec == "c64":
        psi = psi.astype(np.complex64).astype(np.complex128)
    V = rng.uniform(0.5, 2.0, N)
    op = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
    xlo, xhi = 0.123, 3.217  # on no grid point
    o, want = op.observe(xlo, xhi), expected(g, V, psi, xlo, xhi)
    # k-space sums of a complex64 field carry the FP32 transform's rounding (relative
    # error of |phi|^2 summed over N terms: a few 1e-7 times log2 N, averaged)
    tol, ktol = 1e-11, 1e-10 if prec == "c128" else 2e-5
    kmax = max(math.pi * a.n / (a.xmax - a.xmin) for a in (g.x, g.y, g.z))
    for key in ("norm", "energy_v"):
        assert abs(o[key] - want[key]) <= tol * abs(want[key]), key
    assert abs(o["p_range"] - want["p_range"]) <= tol * want["norm"]
    assert abs(o["energy_t"] - want["energy_t"]) <= ktol * max(want["energy_t"], 1e-300)
    assert np.max(np.abs(np.subtract(o["mean_pos"], want["mean_pos"]))) <= tol * 9.0
    assert np.max(np.abs(np.subtract(o["sigma_pos"], want["sigma_pos"]))) <= 1e-6 * 9.0  # a difference of squares
    assert np.max(np.abs(np.subtract(o["mean_mom"], want["mean_mom"]))) <= ktol * kmax
    nrm, peak = op.norm_and_peak()
    assert abs(nrm - want["norm"]) <= tol * want["norm"] and abs(peak - want["peak"]) <= tol * want["peak"]
    assert op.observe(xlo, xhi) == o  # a fixed order: the same bits
    op.close()
