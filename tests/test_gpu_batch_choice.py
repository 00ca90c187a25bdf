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
