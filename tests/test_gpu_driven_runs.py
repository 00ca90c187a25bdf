"""Dipole-driven runs whose kick factors are built in several batches (16 kicks each), and
driven steps with an absorber, against the FP64 oracle taken step by step (the mask after
each step).  Complex128 1e-12 a step, complex64 1e-5 relative L2, as the other driven tests."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AXIS, AMPLITUDE, OMEGA, T0, DT = (0.6, 0.8, 0.3), 0.5, 1.3, 0.1, 0.02


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("mask", [None, "separable", "full"])
@pytest.mark.parametrize("dims,prec", [((36, 20, 15), "c128"), ((36, 20, 15), "c64"), ((64, 32, 1), "c128"),
                                       ((128, 9, 5), "c64"), ((16, 1, 30), "c128")])
def test_runs_across_the_batches_of_kicks(ses, oracle, dims, prec, mask):
    box = tuple(v for d in dims for v in ((-8.0, 8.0) if d > 1 else (0.0, 1.0)))
    live = [1.0 if d > 1 else 0.0 for d in dims]
    V = oracle.harmonic3d(box, dims, 0.8)
    psi = oracle.gaussian3d(box, dims, (1.0, -0.5 * live[1], 0.0), (1.2, 1.2, 1.2), (0.4, 0.0, 0.0))
    g = ses.Grid3D(*(ses.Grid1D(box[2 * a], box[2 * a + 1], dims[a]) for a in range(3)))
    op = ses.SplitOperator3D(g, V, DT, precision=prec)
    m = np.ones(g.size())
    if mask == "separable":
        profiles = [np.linspace(0.98, 1.0, d) for d in dims]
        op.set_absorber_separable(*profiles)
        m = (profiles[0][None, None, :] * profiles[1][None, :, None] * profiles[2][:, None, None]).reshape(-1)
    elif mask == "full":
        m = np.random.default_rng(2).uniform(0.98, 1.0, g.size())
        op.set_absorber(m)
    want, ref = {}, psi
    for i in range(40):
        ref = oracle.driven_step3d(box, dims, V, DT, ref, 1, AXIS, AMPLITUDE, OMEGA, T0 + i * DT) * m
        want[i + 1] = ref
    for steps in (1, 15, 16, 17, 31, 32, 40):
        op.upload_state(psi)
        op.advance_driven(steps, AXIS, AMPLITUDE, OMEGA, T0, absorb=mask is not None)
        assert rel(op.readback(), want[steps]) <= (steps * 1e-12 if prec == "c128" else 1e-5), steps
    op.upload_state(psi)
    done = 0
    for k in (3, 16, 1, 20):  # the same run in several calls
        op.advance_driven(k, AXIS, AMPLITUDE, OMEGA, T0 + done * DT, absorb=mask is not None)
        done += k
    assert rel(op.readback(), want[done]) <= (done * 1e-12 if prec == "c128" else 1e-5)
    op.close()
