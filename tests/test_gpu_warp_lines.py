"""Strided passes with warp-owned lines (every compiled variant, single fields and
batches) against the register path and the FP64 oracle: y and z passes, line counts
that leave the last tile partly empty, more tiles than the ring holds, two-box lines.

Both paths run the same transforms and kinetic arithmetic: 1e-14 (complex128) / 2e-7
(complex64) relative L2 between them, as for the other pipelined passes."""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (dims, precision, first and last warp-line variant of the strided axis)
CASES = [((16, 64, 3), "c64", 1, 1), ((6, 5, 64), "c64", 1, 1), ((16, 64, 3), "c128", 1, 1), ((5, 3, 64), "c128", 1, 1),
         ((16, 128, 3), "c64", 3, 3), ((6, 5, 128), "c64", 3, 3), ((64, 48, 128), "c64", 3, 3),
         ((16, 256, 3), "c64", 4, 4), ((6, 5, 256), "c64", 4, 4), ((256, 256, 9), "c64", 4, 4),
         ((16, 512, 2), "c64", 2, 2), ((10, 3, 512), "c64", 2, 2), ((64, 64, 512), "c64", 2, 2),
         ((16, 128, 3), "c128", 0, 0), ((5, 3, 128), "c128", 0, 0), ((64, 48, 128), "c128", 0, 0),
         ((16, 256, 3), "c128", 3, 3), ((5, 3, 256), "c128", 3, 3), ((128, 256, 5), "c128", 3, 3)]


def scene(ses, oracle, dims):
    box = tuple(v for d in dims for v in ((-7.0, 7.0) if d > 1 else (0.0, 1.0)))
    V = oracle.harmonic3d(box, dims, 0.7)
    psi = oracle.gaussian3d(box, dims, (0.5, 0.4, -0.3), (1.4, 1.3, 1.2), (0.3, -0.2, 0.4))
    g = ses.Grid3D(*(ses.Grid1D(box[2 * a], box[2 * a + 1], dims[a]) for a in range(3)))
    return box, g, V, psi


def make(ses, g, V, psi, prec, svar):
    os.environ["SES_SVAR"], os.environ["SES_PLANE"] = str(svar), "0"
    try:
        return ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
    finally:
        del os.environ["SES_SVAR"], os.environ["SES_PLANE"]


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("dims,prec,first,last", CASES)
def test_warp_lines_match_register_path_and_oracle(ses, oracle, dims, prec, first, last):
    box, g, V, psi = scene(ses, oracle, dims)
    op = make(ses, g, V, psi, prec, -1)
    op.advance(11)
    base = op.readback()
    op.fft3()
    spectrum = op.readback()
    op.close()
    assert rel(base, oracle.step3d(box, dims, V, 0.01, psi, 11)) < (1.1e-11 if prec == "c128" else 1e-5)
    for svar in range(first, last + 1):
        op = make(ses, g, V, psi, prec, svar)
        assert "warp lines" in op.plan_info(), op.plan_info()
        op.advance(11)
        got = op.readback()
        assert rel(got, base) < (1e-14 if prec == "c128" else 2e-7), svar
        op.upload_state(base)
        op.fft3()
        assert rel(op.readback(), spectrum) < (1e-14 if prec == "c128" else 2e-7), svar
        op.fft3(inverse=True)
        assert rel(op.readback(), base) < (1e-14 if prec == "c128" else 1e-6), svar
        op.close()


# more tiles per CTA than the ring holds, on both strided axes
@pytest.mark.parametrize("dims,prec,first,last", [((160, 128, 128), "c64", 3, 3), ((96, 256, 240), "c64", 4, 4),
                                                  ((160, 150, 256), "c64", 4, 4), ((160, 150, 512), "c64", 2, 2),
                                                  ((96, 128, 192), "c128", 0, 0), ((96, 90, 256), "c128", 3, 3),
                                                  ((64, 256, 256), "c128", 3, 3)])
def test_warp_lines_with_rings_in_use(ses, dims, prec, first, last):
    rng = np.random.default_rng(sum(dims))
    g = ses.Grid3D(*(ses.Grid1D(-7.0, 7.0, d) for d in dims))
    V = rng.uniform(0.0, 3.0, g.size())
    psi = rng.standard_normal(g.size()) + 1j * rng.standard_normal(g.size())
    base = None
    for svar in [-1, *range(first, last + 1)]:
        op = make(ses, g, V, psi, prec, svar)
        op.advance(3)
        got = op.readback()
        op.close()
        base = got if base is None else base
        assert rel(got, base) < (1e-14 if prec == "c128" else 2e-7), svar


@pytest.mark.parametrize("dims,prec", [((64, 48, 128), "c64"), ((32, 256, 6), "c64"), ((32, 8, 512), "c64"),
                                       ((32, 24, 128), "c128"), ((32, 16, 256), "c128")])
def test_warp_lines_in_batches(ses, oracle, dims, prec, tmp_path, monkeypatch):
    """Members of one class with their own dt, so their kinetic tables differ, on every
    warp-line variant (chosen through a tune cache)."""
    box, g, V, psi = scene(ses, oracle, dims)
    info = None
    for svar in range(0, 8):
        cache = tmp_path / f"tune{svar}.txt"
        monkeypatch.setenv("SES_TUNE_CACHE", str(cache))
        key = f"sm148:{prec}:batch-s%d:{dims[0]}x{dims[1]}x{dims[2]} {svar}\n"
        cache.write_text("".join(key % q for q in range(3)))
        ops = [ses.SplitOperator3D(g, V, dt, precision=prec, psi0=psi) for dt in (0.01, 0.02, 0.005)]
        with ses.Batch(ops) as b:
            b.step(10)
            info = b.info()
            b.sync()
            for op, dt in zip(ops, (0.01, 0.02, 0.005)):
                want = oracle.step3d(box, dims, V, dt, psi, 10)
                assert rel(op.readback(), want) < (1e-11 if prec == "c128" else 1e-5), (svar, dt, info)
        for op in ops:
            op.close()


def test_expired_wait_in_a_warp_line_pass(ses, oracle):
    """The failure-detection hook on a warp-line pass: the wait runs out (1 ms, 16 bytes
    that no copy delivers), the status says so, and the handle steps correctly after."""
    dims = (16, 16, 256)
    box, g, V, psi = scene(ses, oracle, dims)
    op = make(ses, g, V, psi, "c64", 4)
    op.set_wait_limit(2_000_000, 16)
    op.advance(2)
    with pytest.raises(TimeoutError):
        op.sync(30000)
    op.set_wait_limit(0, 0)
    op.upload_state(psi)
    op.advance(5)
    assert rel(op.readback(), oracle.step3d(box, dims, V, 0.01, psi, 5)) < 1e-5
    op.close()
