"""Contiguous passes on staged rows (the default of most lengths) against the register
path and the FP64 oracle: every compiled length, line counts that leave the last tile
partly empty or fill one tile only, no absorber, a separable one and a full array.

Both paths run the same transforms and diagonal arithmetic: 1e-14 (complex128) /
2e-7 (complex64) relative L2 between them, as for the pipelined passes."""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(16, 3, 5), (32, 6, 3), (48, 5, 4), (64, 1, 9), (96, 9, 2), (128, 3, 3), (160, 5, 5), (256, 3, 5), (512, 5, 2),
        (1024, 3, 1)]


def run(ses, g, V, psi, prec, xvar, mask):
    os.environ["SES_XVAR"], os.environ["SES_PLANE"] = str(xvar), "0"
    try:
        op = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
    finally:
        del os.environ["SES_XVAR"], os.environ["SES_PLANE"]
    info = op.plan_info()
    op.set_absorber(mask)
    op.advance(11, absorb=True)
    out = op.readback()
    op.close()
    return out, info


@pytest.mark.parametrize("prec", ["c128", "c64"])
@pytest.mark.parametrize("dims", DIMS, ids=["x".join(map(str, d)) for d in DIMS])
def test_staged_rows_match_register_path_and_oracle(ses, oracle, dims, prec):
    box = tuple(v for d in dims for v in ((-7.0, 7.0) if d > 1 else (0.0, 1.0)))
    live = [1.0 if d > 1 else 0.0 for d in dims]
    V = oracle.harmonic3d(box, dims, 0.7)
    psi = oracle.gaussian3d(box, dims, tuple(0.5 * a for a in live), (1.4, 1.3, 1.2), tuple(0.3 * a for a in live))
    g = ses.Grid3D(*(ses.Grid1D(box[2 * a], box[2 * a + 1], dims[a]) for a in range(3)))
    sep = oracle.mask3d(box, dims, 1.5, 1)
    full = sep * (1.0 - 0.01 * np.random.default_rng(3).random(sep.size))
    for mask in (None, sep, full):
        a, ia = run(ses, g, V, psi, prec, 64, mask)
        b, ib = run(ses, g, V, psi, prec, -1, mask)
        assert "staged rows" not in ib
        if not (prec == "c128" and dims[0] == 1024):  # 1024 has a compiled plan in complex64 only
            assert "staged rows" in ia, ia
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < (1e-14 if prec == "c128" else 2e-7)
        want = oracle.step3d(box, dims, V, 0.01, psi, 11, mask=mask)
        assert np.linalg.norm(a - want) / np.linalg.norm(want) < (1.1e-11 if prec == "c128" else 1e-5)
