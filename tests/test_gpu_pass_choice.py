"""The kernels that a handle's passes run on by default: by axis length, precision and
the number of lines of the pass, reported by plan_info as they are launched, and the same
results whichever kernel a pass runs on.

Tolerances between two kernels of one pass and against the FP64 oracle are those of the
suite: 1e-14 (complex128) / 2e-7 (complex64) and 1e-12 a step / 1e-5 relative L2."""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def plain_environment(monkeypatch, tmp_path):
    for name in ("SES_XVAR", "SES_SVAR", "SES_PIPELINED", "SES_LONG"):
        monkeypatch.delenv(name, raising=False)
    monkeypatch.setenv("SES_TUNE_CACHE", str(tmp_path / "none.txt"))
    monkeypatch.setenv("SES_PLANE", "0")


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def grid(ses, dims):
    return ses.Grid3D(*(ses.Grid1D(-7.0, 7.0, d) if d > 1 else ses.Grid1D(0.0, 1.0, 1) for d in dims))


def scene(ses, dims, seed=0):
    rng = np.random.default_rng([seed, *dims])
    g = grid(ses, dims)
    return g, rng.uniform(0.0, 3.0, g.size()), rng.standard_normal(g.size()) + 1j * rng.standard_normal(g.size())


def parts(op):
    return dict(zip("xyz", op.plan_info().split("; ")[:3]))


# ---- first and last x passes of a call ----

X_VARIANTS = [(32, "c64", False), (48, "c64", False), (64, "c64", True), (96, "c64", True), (128, "c64", True),
              (160, "c64", True), (256, "c64", True), (512, "c64", True), (1024, "c64", False), (32, "c128", False),
              (64, "c128", True), (96, "c128", False), (128, "c128", False), (256, "c128", True), (512, "c128", True)]


@pytest.mark.parametrize("nx,prec,fed", X_VARIANTS)
def test_first_and_last_x_passes(ses, nx, prec, fed):
    """They run on the TMA-fed kernel where one is built (a one-step call of 256^3 complex64
    takes 296 us so, 448 without), and a run split into calls gives the bits of one call."""
    dims = (nx, 32, 25 if nx < 512 else 9)
    g, V, psi = scene(ses, dims)
    op = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
    x = parts(op)["x"]
    assert ("pipelined" in x) == fed, x
    profiles = [np.linspace(0.97, 1.0, d) for d in dims]
    full = np.random.default_rng(1).uniform(0.97, 1.0, g.size())
    for mask in (None, "separable", "full"):
        if mask == "separable":
            op.set_absorber_separable(*profiles)
        elif mask == "full":
            op.set_absorber(full)
        outs = []
        for split in ((6,), (1, 1, 1, 1, 1, 1), (2, 4)):
            op.upload_state(psi)
            for k in split:
                op.advance(k, absorb=mask is not None)
            outs.append(op.readback())
        assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2]), mask
    op.close()


@pytest.mark.parametrize("nx,prec", [(64, "c64"), (96, "c64"), (128, "c64"), (160, "c64"), (256, "c64"), (64, "c128"),
                                     (128, "c128")])
def test_batches_split_into_calls_and_mixed_absorbers(ses, oracle, nx, prec):
    """Members without an absorber, with a separable one and with a full one: all of a class
    alike, and mixed."""
    dims = (nx, 32, 32)
    g, V, psi = scene(ses, dims)
    profiles = [np.linspace(0.97, 1.0, d) for d in dims]
    sep = (profiles[0][None, None, :] * profiles[1][None, :, None] * profiles[2][:, None, None]).reshape(-1)
    full = np.random.default_rng(1).uniform(0.97, 1.0, g.size())
    tol = 6e-12 if prec == "c128" else 1e-5
    want = {m: oracle.step3d(g.box, dims, V, 0.01, psi, 6, mask=v) for m, v in (("n", None), ("s", sep), ("f", full))}
    for members in ("nn", "ss", "ff", "nsf", "sf"):
        ops = []
        for m in members:
            op = ses.SplitOperator3D(g, V, 0.01, precision=prec)
            if m == "s":
                op.set_absorber_separable(*profiles)
            elif m == "f":
                op.set_absorber(full)
            ops.append(op)
        with ses.Batch(ops) as b:
            assert "member-by-member" not in b.info(), b.info()
            first = None
            for split in ((6,), (1, 1, 1, 3)):
                for op in ops:
                    op.upload_state(psi)
                for k in split:
                    b.step(k, absorb=True)
                b.sync()
                outs = [op.readback() for op in ops]
                first = first or outs
                assert all(np.array_equal(a, c) for a, c in zip(first, outs)), members
        for m, out in zip(members, first):
            assert rel(out, want[m]) < tol, (members, m)
        for op in ops:
            op.close()


# ---- defaults by the number of lines ----

# (axis, dims with few lines, dims with more, precision, text of the first, text of the second)
BY_LINES = [("y", (64, 512, 1), (64, 512, 40), "c64", "register-path", "TMA lines=8"),
            ("z", (16, 128, 512), (32, 72, 512), "c64", "register-path", "warp lines=8"),
            ("z", (64, 64, 256), (64, 72, 256), "c64", "TMA lines=8", "warp lines=8"),
            ("y", (64, 256, 64), (64, 256, 65 + 7), "c64", "TMA lines=8", "warp lines=8"),
            ("z", (64, 128, 128), (96, 96, 128), "c64", "TMA lines=8", "warp lines=16"),
            ("z", (64, 128, 128), (96, 96, 128), "c128", "register-path", "warp lines=8"),
            ("y", (128, 128, 64), (128, 128, 72), "c128", "register-path", "warp lines=8"),
            ("y", (256, 256, 1), (64, 256, 36), "c128", "TMA lines=4", "warp lines=4"),
            ("z", (32, 64, 256), (36, 64, 256), "c128", "TMA lines=4", "warp lines=4"),
            ("x", (256, 512, 1), (256, 540, 1), "c128", "pipelined warps=2", "staged rows"),
            ("x", (512, 256, 1), (512, 270, 1), "c128", "pipelined warps=2", "staged rows")]


@pytest.mark.parametrize("axis,few,more,prec,t_few,t_more", BY_LINES)
def test_defaults_follow_the_number_of_lines(ses, axis, few, more, prec, t_few, t_more):
    for dims, text in ((few, t_few), (more, t_more)):
        g, V, psi = scene(ses, dims)
        op = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
        assert text in parts(op)[axis], (dims, op.plan_info())
        op.advance(3)
        got = op.readback()
        op.close()
        os.environ["SES_XVAR"] = os.environ["SES_SVAR"] = "-1"
        op = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
        del os.environ["SES_XVAR"], os.environ["SES_SVAR"]
        assert "pipelined" not in op.plan_info() and "staged" not in op.plan_info()
        op.advance(3)
        assert rel(got, op.readback()) < (1e-14 if prec == "c128" else 2e-7), dims
        op.close()


@pytest.mark.parametrize("dims,prec,form", [((64, 64, 64), "c64", "2 CTAs"), ((64, 64, 96), "c64", "1 CTA "),
                                            ((96, 96, 64), "c64", "four"), ((96, 96, 128), "c64", "1 CTA "),
                                            ((96, 96, 192), "c64", "four"), ((64, 64, 64), "c128", "2 CTAs")])
def test_step_form_follows_the_number_of_planes(ses, oracle, dims, prec, form, monkeypatch):
    monkeypatch.delenv("SES_PLANE")
    g, V, psi = scene(ses, dims)
    op = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
    assert form in op.plan_info(), op.plan_info()
    op.advance(4)
    assert rel(op.readback(), oracle.step3d(g.box, dims, V, 0.01, psi, 4)) < (4e-12 if prec == "c128" else 1e-5)
    op.close()


# ---- run-time plans with few lines along y or z: tiles of 1, 2 and 4 lines ----

NARROW = [(64, 1536, 1), (5, 1500, 1), (128, 1000, 1), (256, 300, 1), (100, 2048, 1), (256, 4096, 1), (512, 1000, 1),
          (512, 1536, 1), (20, 1000, 8), (9, 15, 1080), (3, 2, 2000), (1, 27, 750), (250, 1, 600)]


@pytest.mark.parametrize("prec", ["c64", "c128"])
@pytest.mark.parametrize("dims", NARROW, ids=["x".join(map(str, d)) for d in NARROW])
def test_narrow_tiles(ses, oracle, dims, prec):
    g, V, psi = scene(ses, dims)
    op = ses.SplitOperator3D(g, V, 0.01, precision=prec, psi0=psi)
    op.advance(3)
    assert rel(op.readback(), oracle.step3d(g.box, dims, V, 0.01, psi, 3)) < (3e-12 if prec == "c128" else 1e-5)
    op.upload_state(psi)
    op.fft3()
    want = np.fft.fftn(psi.reshape(g.shape)).reshape(-1)
    assert rel(op.readback(), want) < (1e-14 if prec == "c128" else 5e-7) * np.log2(g.size())
    op.close()


# ---- what plan_info says ----

@pytest.mark.parametrize("prec", ["c64", "c128"])
def test_plan_info_names_the_kernels_that_run(ses, prec, monkeypatch):
    g, V, psi = scene(ses, (128, 1, 1))
    op = ses.SplitOperator3D(g, V, 0.01, precision=prec)  # a line steps on the run-time plan's kernel
    assert "run-time plan" in op.plan_info() and "staged" not in op.plan_info(), op.plan_info()
    op.close()
    line = ses.line_grid(ses.Grid1D(-7.0, 7.0, 24576))  # no cluster: two register-path launches a step
    op = ses.SplitOperator3D(line, np.zeros(24576), 0.01, precision=prec)
    assert "staged" not in op.plan_info() and "pipelined" not in op.plan_info(), op.plan_info()
    op.close()
    g, V, psi = scene(ses, (100, 128, 72))  # x has no compiled plan, and 100 is no multiple of a y tile's lines
    op = ses.SplitOperator3D(g, V, 0.01, precision="c64")
    monkeypatch.setenv("SES_SVAR", "0")
    forced = ses.SplitOperator3D(g, V, 0.01, precision="c64")
    assert "register-path" in parts(forced)["y"], forced.plan_info()
    op.close()
    forced.close()
    monkeypatch.setenv("SES_PIPELINED", "0")
    g, V, psi = scene(ses, (128, 128, 72))
    op = ses.SplitOperator3D(g, V, 0.01, precision=prec)
    assert "staged" not in op.plan_info() and "pipelined" not in op.plan_info(), op.plan_info()
    op.close()
