"""Long 1D lines stepped by one thread-block cluster (SES_LONG unset or its CTA count)
against the two-launch form (SES_LONG=0) and the FP64 oracle: every compiled line,
with and without an absorber, one step and runs split over calls.

The two forms run the same plans and diagonal arithmetic in differently structured
kernels: they agree to 1e-14 (complex128) / 2e-7 (complex64) relative L2, as the step
forms of 3D grids; within the cluster form a split run gives the same bits."""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(8192, "c64", 8), (8192, "c128", 8), (16384, "c64", 8), (16384, "c128", 8), (32768, "c64", 16),
         (32768, "c64", 8), (32768, "c128", 16), (32768, "c128", 8), (65536, "c64", 16), (65536, "c64", 8),
         (65536, "c128", 16), (131072, "c64", 16)]


def run(ses, g, V, psi, prec, form, parts, mask=None):
    os.environ["SES_LONG"] = str(form)
    try:
        op = ses.SplitOperator3D(g, V, 0.002, precision=prec, psi0=psi)
    finally:
        del os.environ["SES_LONG"]
    info = op.plan_info()
    if mask is not None:
        op.set_absorber(mask)
    for k in parts:
        op.advance(k, absorb=mask is not None)
    out = op.readback()
    op.close()
    return out, info


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n,prec,cs", CASES)
def test_cluster_line_matches_two_launches_and_oracle(ses, oracle, n, prec, cs):
    g = ses.line_grid(ses.Grid1D(-60.0, 60.0, n))
    x = np.asarray(g.x.coords())
    V = 0.02 * x * x
    psi = oracle.gaussian3d(g.box, g.dims, (1.5, 0.0, 0.0), (1.2, 1.0, 1.0), (0.6, 0.0, 0.0))
    mask = np.clip((60.0 - np.abs(x)) / 6.0, 0.0, 1.0) ** 0.125 * (1.0 - 0.01 * (np.arange(n) % 7 == 3))
    for m in (None, mask):
        for parts in ((1,), (12,)):
            a, ia = run(ses, g, V, psi, prec, cs, parts, m)
            b, ib = run(ses, g, V, psi, prec, 0, parts, m)
            assert f"cluster of {cs} CTAs" in ia and "cluster" not in ib, (ia, ib)
            assert rel(a, b) < (1e-14 if prec == "c128" else 2e-7), (parts, rel(a, b))
    want = oracle.step3d(g.box, g.dims, V, 0.002, psi, 12, mask=mask)
    assert rel(a, want) < (1.2e-11 if prec == "c128" else 1e-5)
    split, _ = run(ses, g, V, psi, prec, cs, (3, 1, 8), mask)
    assert np.array_equal(split, a)
