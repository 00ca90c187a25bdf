"""The kernels a batch class runs on: a selection given to its first member, warp-line
variants chosen through the tune cache, and 1D lines alone and in batches.

Tolerances: complex128 1e-12 a step, complex64 1e-5 relative L2 against the oracle, and
twice that between two plans of one line."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def plain_environment(monkeypatch, tmp_path):
    for name in ("SES_XVAR", "SES_SVAR", "SES_PIPELINED", "SES_PLANE", "SES_BATCH_PLANE"):
        monkeypatch.delenv(name, raising=False)
    monkeypatch.setenv("SES_TUNE_CACHE", str(tmp_path / "none.txt"))


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def scene(ses, oracle, dims):
    box = tuple(v for d in dims for v in ((-7.0, 7.0) if d > 1 else (0.0, 1.0)))
    V = oracle.harmonic3d(box, dims, 0.7)
    psi = oracle.gaussian3d(box, dims, (0.5, 0.4, -0.3), (1.4, 1.3, 1.2), (0.3, -0.2, 0.4))
    return ses.Grid3D(*(ses.Grid1D(box[2 * a], box[2 * a + 1], dims[a]) for a in range(3))), V, psi


def sm_count():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("by", ["environment", "cache"])
def test_a_members_selection_reaches_its_class(ses, oracle, by, monkeypatch, tmp_path):
    dims = (128, 32, 64)
    g, V, psi = scene(ses, oracle, dims)
    if by == "environment":
        monkeypatch.setenv("SES_XVAR", "0")
        monkeypatch.setenv("SES_SVAR", "0")
    else:
        cache = tmp_path / "tune.txt"
        rows = ((0, "x"), (1, "s"), (2, "fused"))
        cache.write_text("".join(f"sm{sm_count()}:c64:{r}:{dims[a]}:{g.size() // dims[a]} 0\n" for a, r in rows))
        monkeypatch.setenv("SES_TUNE_CACHE", str(cache))
    ops = [ses.SplitOperator3D(g, V, dt, precision="c64", psi0=psi) for dt in (0.01, 0.02)]
    with ses.Batch(ops) as b:
        assert all(f"{p}=pipe0" in b.info() for p in ("x", "s0", "s1", "s2")), b.info()
        b.step(10)
        b.sync()
        for op, dt in zip(ops, (0.01, 0.02)):
            assert rel(op.readback(), oracle.step3d(g.box, dims, V, dt, psi, 10)) < 1e-5
    for op in ops:
        op.close()


# (dims, precision, warp-line variant, strided passes that it serves)
WARP = [((64, 64, 32), "c64", 1, "02"), ((32, 32, 64), "c64", 1, "1"), ((32, 128, 32), "c64", 3, "02"),
        ((64, 48, 128), "c64", 3, "1"), ((32, 256, 32), "c64", 4, "02"), ((32, 32, 256), "c64", 4, "1"),
        ((32, 512, 32), "c64", 2, "02"), ((32, 32, 512), "c64", 2, "1"), ((32, 64, 32), "c128", 1, "02"),
        ((32, 32, 64), "c128", 1, "1"), ((32, 128, 32), "c128", 0, "02"), ((32, 48, 128), "c128", 0, "1"),
        ((32, 256, 32), "c128", 3, "02"), ((48, 32, 256), "c128", 3, "1"), ((128, 256, 1), "c64", 4, "0"),
        ((64, 128, 1), "c128", 0, "0")]


@pytest.mark.parametrize("dims,prec,svar,passes", WARP)
def test_warp_lines_run_in_batches(ses, oracle, dims, prec, svar, passes, monkeypatch, tmp_path):
    """Members with their own dt, so their kinetic tables differ, on the batched warp-line
    kernels, which the class reports."""
    g, V, psi = scene(ses, oracle, dims)
    cache = tmp_path / "tune.txt"
    cache.write_text("".join(f"sm{sm_count()}:{prec}:batch-s{q}:{dims[0]}x{dims[1]}x{dims[2]} {svar}\n" for q in passes))
    monkeypatch.setenv("SES_TUNE_CACHE", str(cache))
    dts = (0.01, 0.02, 0.005)
    ops = [ses.SplitOperator3D(g, V, dt, precision=prec, psi0=psi) for dt in dts]
    with ses.Batch(ops) as b:
        assert all(f"s{q}=pipe{svar}" in b.info() for q in passes), b.info()
        b.step(10)
        b.sync()
        for op, dt in zip(ops, dts):
            want = oracle.step3d(g.box, dims, V, dt, psi, 10)
            assert rel(op.readback(), want) < (1e-11 if prec == "c128" else 1e-5), dt
    for op in ops:
        op.close()


@pytest.mark.parametrize("prec", ["c64", "c128"])
@pytest.mark.parametrize("n", [64, 128, 512, 1024])
def test_lines_alone_and_in_a_batch(ses, oracle, n, prec):
    """A line alone steps on the run-time plan, a batch of compiled lengths on theirs: the
    same step to rounding."""
    g, V, psi = scene(ses, oracle, (n, 1, 1))
    alone = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
    alone.advance(10)
    ops = [ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi) for _ in range(2)]
    with ses.Batch(ops) as b:
        b.step(10)
        b.sync()
        got = [op.readback() for op in ops]
    assert np.array_equal(got[0], got[1])
    assert rel(alone.readback(), got[0]) < (2e-11 if prec == "c128" else 2e-5)
    want = oracle.step3d(g.box, g.dims, V, 0.01, psi, 10)
    assert rel(got[0], want) < (1e-11 if prec == "c128" else 1e-5)
    for op in (alone, *ops):
        op.close()
