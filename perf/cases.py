"""The work this framework is timed on, each case through the public Python surface.

A case is one scene on one grid: the state holds a solver handle (or a batch of
them) with its potential, absorber and packet resident on the device, as a
program keeps it between calls; a pass advances it and reads what that program
reads -- the observables, or a frame's density slice and norm.  The field
evolves from pass to pass.

Grids, time steps, absorbers and cadences are those of the repository's own
workloads (scenes.py, bench.py) and tests.  Potentials and packets are drawn
from the seed inside the ranges those workloads use.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import shoeridingerequationsolver_b200 as ses

PI = math.pi
SWEEP_SIZES = (32, 48, 64, 96, 128, 160)  # the batched sweep's


def listed():
    return [
        # the smallest calls: a 1D textbook scene, a few steps between plots
        dict(name="line_1024_c128", kind="steps", scene="well", nx=1024, ny=1, nz=1, precision="c128", steps=10,
             absorb=False),
        # an interactive frame: some steps, the density slice that is drawn, the norm that is watched
        dict(name="frame_64_c64", kind="frame", scene="coulomb", nx=64, ny=64, nz=64, precision="c64", steps=8,
             absorb=True),
        # plain FP64 harmonic trap, observed every 100 steps
        dict(name="trap_64_c128", kind="steps", scene="trap", nx=64, ny=64, nz=64, precision="c128", steps=100,
             absorb=False),
        # a relaxation to the ground state, renormalised after every step (the reference's default)
        dict(name="relax_64_c128", kind="relax", scene="trap", nx=64, ny=64, nz=64, precision="c128", steps=50,
             absorb=False),
        # a served 1D request: a long line, observed every 100 steps
        dict(name="line_65536_c64", kind="steps", scene="well", nx=65536, ny=1, nz=1, precision="c64", steps=100,
             absorb=True),
        # a served 2D request: the stadium billiard, observed every 100 steps
        dict(name="plane_1024_c64", kind="steps", scene="stadium", nx=1024, ny=1024, nz=1, precision="c64", steps=100,
             absorb=True),
        # an atom in a laser field: the dipole drive, every step with its own kick
        dict(name="driven_128_c64", kind="driven", scene="coulomb", nx=128, ny=128, nz=128, precision="c64", steps=20,
             absorb=True),
        # a box that is no cube, with lengths that are no powers of two
        dict(name="ragged_120x100x90_c128", kind="steps", scene="trap", nx=120, ny=100, nz=90, precision="c128",
             steps=50, absorb=True),
        # the batched tunnelling sweep: many independent instances of mixed sizes
        dict(name="sweep_36_c64", kind="batch", scene="barrier", sizes=",".join(map(str, SWEEP_SIZES)), count=36,
             precision="c64", steps=30, absorb=True),
        # Coulomb + Stark with an absorber, in both precisions
        dict(name="coulomb_256_c64", kind="steps", scene="coulomb", nx=256, ny=256, nz=256, precision="c64", steps=100,
             absorb=True),
        dict(name="coulomb_256_c128", kind="steps", scene="coulomb", nx=256, ny=256, nz=256, precision="c128",
             steps=50, absorb=True),
        # the largest: tunnelling on 512^3, the transmitted probability every 50 steps
        dict(name="tunnel_512_c64", kind="steps", scene="barrier", nx=512, ny=512, nz=512, precision="c64", steps=50,
             absorb=True),
    ]


def _lengths(lo, hi):
    """Every axis length 2^a 3^b 5^c in [lo, hi], odd ones among them."""
    out = set()
    for a in range(13):
        for b in range(8):
            for c in range(6):
                n = 2 ** a * 3 ** b * 5 ** c
                if lo <= n <= hi:
                    out.add(n)
    return sorted(out)


def _length(rng, lo, hi):
    """One supported length, log-uniform over [lo, hi]; a power of two half of the time."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    some = [n for n in _lengths(lo, hi) if n & (n - 1) == 0] if rng.random() < 0.5 else _lengths(lo, hi)
    return min(some, key=lambda n: abs(math.log(n / want)))


def draw(rng):
    precision = rng.choice(["c64", "c128"])
    absorb = rng.random() < 0.6
    kind = rng.choice(["line", "plane", "box", "box", "cube", "cube", "frame", "relax", "driven", "batch"])
    if kind == "batch":
        sizes = sorted({_length(rng, 24, 160) for _ in range(rng.randint(1, 4))})
        points = sum(n ** 3 for n in sizes)
        count = max(len(sizes), min(48, int(len(sizes) * 3e7 / points)))
        return dict(kind="batch", scene="barrier", sizes=",".join(map(str, sizes)), count=rng.randint(len(sizes), count),
                    precision=precision, steps=rng.randint(5, 50), absorb=absorb)
    if kind == "line":
        nx = rng.choice([8192, 16384, 32768, 65536, 131072, 262144]) if rng.random() < 0.4 else _length(rng, 256, 4096)
        return dict(kind="steps", scene="well", nx=nx, ny=1, nz=1, precision=precision, steps=rng.randint(5, 200),
                    absorb=absorb)
    if kind == "plane":
        return dict(kind="steps", scene=rng.choice(["stadium", "trap"]), nx=_length(rng, 64, 2048),
                    ny=_length(rng, 64, 2048), nz=1, precision=precision, steps=rng.randint(5, 100), absorb=absorb)
    if kind == "box":
        dims = [_length(rng, 24, 320) for _ in range(3)]
    else:
        dims = [_length(rng, 32, 320 if kind == "cube" else 160)] * 3
    points = dims[0] * dims[1] * dims[2]
    most = max(5, min(100, int(1.5e9 / points)))
    scene = "trap" if kind == "relax" else rng.choice(["trap", "coulomb", "barrier"])
    return dict(kind=kind if kind in ("frame", "relax", "driven") else "steps", scene=scene, nx=dims[0], ny=dims[1],
                nz=dims[2], precision=precision, steps=rng.randint(4, 16) if kind == "frame" else rng.randint(5, most),
                absorb=absorb and kind != "relax")


# ---- the scenes: potential, packet, absorber, on the device, from the seed alone ----

DT = {"trap": 0.005, "coulomb": 0.01, "barrier": 0.002, "stadium": 0.005, "well": 0.005}


def _half(scene, n):
    """Half the box along an axis of n points (a collapsed axis is [0, 1))."""
    if scene == "trap":
        return 10.0
    if scene == "coulomb":
        return 0.15625 * n   # spacing 0.3125: [-40, 40) at 256
    if scene == "barrier":
        return 0.1171875 * n  # spacing 0.234: [-60, 60) at 512
    if scene == "stadium":
        return 30.0
    return 200.0 if n > 4096 else 25.0


class _Scene:
    """One instance on an nx x ny x nz grid: axes, V and psi0 as FP64 device arrays [z, y, x], mask profiles."""

    def __init__(self, scene, dims, rng, dt=None):
        self.dims, self.dt = dims, dt or DT[scene]
        self.box = []
        for n in dims:
            self.box += [-_half(scene, n), _half(scene, n)] if n > 1 else [0.0, 1.0]
        self.h = [(self.box[2 * a + 1] - self.box[2 * a]) / dims[a] for a in range(3)]
        self.r = [self.box[2 * a] + self.h[a] * torch.arange(dims[a], dtype=torch.float64, device="cuda")
                  for a in range(3)]
        self.x, self.y, self.z = self.r[0][None, None, :], self.r[1][None, :, None], self.r[2][:, None, None]
        shape = dims[::-1]
        live = [1.0 if n > 1 else 0.0 for n in dims]
        x, y, z = self.x, self.y, self.z
        if scene == "trap":
            c = rng.uniform(-0.5, 0.5, 3) * live
            v = 0.5 * rng.uniform(0.5, 1.5) ** 2 * ((x - c[0]) ** 2 + live[1] * (y - c[1]) ** 2
                                                     + live[2] * (z - c[2]) ** 2)
            packets = [(rng.uniform(-2.0, 2.0, 3), rng.uniform(0.8, 1.4, 3), rng.uniform(-0.5, 0.5, 3))]
        elif scene == "coulomb":
            rad = torch.sqrt(x * x + y * y + z * z)
            near = 1e-6 * self.h[0]
            v = torch.where(rad < near, -2.3800774 / self.h[0], -1.0 / torch.clamp(rad, min=near))
            v = v + rng.uniform(0.0, 0.02) * z
            packets = [(rng.uniform(-3.0, 3.0, 3), np.full(3, rng.uniform(0.8, 2.0)), np.zeros(3)) for _ in range(4)]
        elif scene == "barrier":
            v = torch.where((x >= -1.0) & (x < 1.0), rng.uniform(0.5, 5.0), 0.0)
            s = np.full(3, rng.uniform(1.0, 2.5))
            packets = [(np.array([0.33 * self.box[0], 0.0, 0.0]), s, np.array([rng.uniform(1.0, 4.0), 0.0, 0.0]))]
        elif scene == "stadium":
            inside = x - torch.clamp(x, -6.5, 6.5)
            v = torch.where(torch.sqrt(inside * inside + y * y) > 13.0, 50.0, 0.0)
            packets = [(rng.uniform(-2.0, 2.0, 3), np.full(3, rng.uniform(1.0, 2.0)),
                        np.append(rng.uniform(-2.0, 2.0, 2), 0.0))]
        else:  # "well": Morse
            q = 1.0 - torch.exp(-0.5 * x)
            v = torch.clamp(rng.uniform(0.5, 10.0) * q * q, max=1e3)
            packets = [(rng.uniform(-0.5, 0.5, 3), np.full(3, rng.uniform(0.8, 1.2)), rng.uniform(0.2, 0.8, 3))]
        self.v = v.expand(shape).contiguous()
        psi = torch.zeros(shape, dtype=torch.complex128, device="cuda")
        for c, s, k in packets:
            parts = [torch.exp(-((self.r[a] - live[a] * c[a]) ** 2) / (4.0 * s[a] * s[a])
                               + 1j * live[a] * k[a] * self.r[a]) for a in range(3)]
            psi += np.exp(1j * rng.uniform(0.0, 2.0 * PI)) * (
                parts[0][None, None, :] * parts[1][None, :, None] * parts[2][:, None, None])
        self.dv = self.h[0] * self.h[1] * self.h[2]
        self.psi = psi / torch.sqrt(psi.abs().square().sum() * self.dv)
        self.mask = []  # cos^(1/8) ramp on the outer 10% of each axis
        for a in range(3):
            if dims[a] == 1:
                self.mask.append(np.ones(1))
                continue
            lo, hi = self.box[2 * a], self.box[2 * a + 1]
            u = lo + self.h[a] * np.arange(dims[a])
            d, width = np.minimum(u - lo, hi - u), 0.1 * (hi - lo)
            m = np.power(np.sin(0.5 * PI * np.minimum(d, width) / width), 0.125)
            self.mask.append(np.where(d >= width, 1.0, m))

    def grid(self):
        return ses.Grid3D(*(ses.Grid1D(self.box[2 * a], self.box[2 * a + 1], self.dims[a]) for a in range(3)))


def _scenes(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        sizes = [int(n) for n in case["sizes"].split(",")]
        for i in range(case["count"]):
            yield _Scene(case["scene"], (sizes[i % len(sizes)],) * 3, rng, dt=0.005)
    else:
        yield _Scene(case["scene"], (case["nx"], case["ny"], case["nz"]), rng)


PAST = 1.003  # x beyond which the packet counts as transmitted (on no grid point, where rounding would decide)
DRIVE = dict(axis=(0.6, 0.0, 0.8), amplitude=0.05, omega=0.6)  # field polarisation, strength, frequency


class _DeviceField:
    """The resident psi as an array torch can wrap; it holds the handle that owns the memory."""

    def __init__(self, op, precision):
        self.op = op
        ptr, _ = op.psi_device()
        self.__cuda_array_interface__ = dict(shape=op.grid.shape, typestr="<c8" if precision == "c64" else "<c16",
                                             data=(ptr, False), version=3, strides=None)


def prepare(case, seed):
    ops, fields = [], []
    for s in _scenes(case, seed):
        make = ses.ImaginaryTimePropagator3D if case["kind"] == "relax" else ses.SplitOperator3D
        op = make(s.grid(), s.v.cpu().numpy().reshape(-1), s.dt, precision=case["precision"])
        if case["absorb"]:
            op.set_absorber_separable(*s.mask)
        field = torch.as_tensor(_DeviceField(op, case["precision"]), device="cuda")
        field.copy_(s.psi)
        ops.append(op)
        fields.append(field)
    torch.cuda.synchronize()
    state = dict(case=case, ops=ops, fields=fields)
    if case["kind"] == "batch":
        state["batch"] = ses.Batch(ops)
    return state


def _readings(values, case):
    """FP64 readings of an FP64 run; of a complex64 run, to the precision its field has."""
    return np.array(values, dtype=np.float64 if case["precision"] == "c128" else np.float32)


def _row(o):
    return [o["norm"], o["energy"], o["energy_v"], o["energy_t"], o["p_range"], *o["mean_pos"], *o["sigma_pos"],
            *o["mean_mom"]]


def run(state):
    case, ops = state["case"], state["ops"]
    kind, steps, absorb = case["kind"], case["steps"], case["absorb"]
    if kind == "batch":
        state["batch"].step(steps, absorb=absorb)
        rows = state["batch"].observe(PAST, math.inf)
        return dict(psi=state["fields"], readings=_readings([_row(o) for o in rows], case))
    op, psi = ops[0], state["fields"][0]
    if kind == "relax":
        return dict(psi=psi, readings=_readings([op.relax_resident(steps)], case))
    if kind == "driven":
        op.advance_driven(steps, DRIVE["axis"], DRIVE["amplitude"], DRIVE["omega"], absorb=absorb)
    else:
        op.advance(steps, absorb=absorb)
    if kind == "frame":
        density = op.density_slice(2, case["nz"] // 2)
        return dict(psi=psi, density=density, readings=_readings(op.norm_and_peak(), case))
    return dict(psi=psi, readings=_readings(_row(op.observe(PAST, math.inf)), case))


def work(case):
    """Bytes and operations one pass cannot do without.

    Every step transforms the whole field forward and back (5 N log2 N each) and
    multiplies it by two phases (and the absorber).  A field that the chip's 126 MB
    cache cannot hold is read and written, and its potential phase read, once a
    step; a smaller one once a pass.  The readings take one more transform and one
    more pass over field and potential."""
    esize = 16 if case["precision"] == "c128" else 8
    if case["kind"] == "batch":
        sizes = [int(n) for n in case["sizes"].split(",")]
        grids = [(sizes[i % len(sizes)],) * 3 for i in range(case["count"])]
    else:
        grids = [(case["nx"], case["ny"], case["nz"])]
    points = [g[0] * g[1] * g[2] for g in grids]
    held = sum(points) * 2 * esize <= 126e6
    out = dict(bytes=0, flops=0)
    for n in points:
        transform = 5.0 * n * math.log2(n)
        out["flops"] += case["steps"] * (2 * transform + (14 if case["absorb"] else 12) * n)
        out["bytes"] += (1 if held else case["steps"]) * 3 * esize * n
        if case["kind"] not in ("frame", "relax"):
            out["flops"] += transform + 30 * n
            out["bytes"] += (esize + 8) * n
    return out


# ---- the same in 64 bits, in plain torch ----

def _wavenumbers(s):
    return [2.0 * PI * torch.fft.fftfreq(s.dims[a], s.h[a], dtype=torch.float64, device="cuda") for a in range(3)]


def _exact_row(s, psi):
    w = psi.abs().square()
    k = _wavenumbers(s)
    phi = torch.fft.fftn(psi).abs().square()
    total, ktotal = w.sum(), phi.sum()
    along = [w.sum((0, 1)), w.sum((0, 2)), w.sum((1, 2))]
    kalong = [phi.sum((0, 1)), phi.sum((0, 2)), phi.sum((1, 2))]
    ev = (s.v * w).sum() / total
    et = sum((0.5 * k[a] * k[a] * kalong[a]).sum() for a in range(3)) / ktotal
    mean = [(s.r[a] * along[a]).sum() / total for a in range(3)]
    sigma = [torch.sqrt(torch.clamp((s.r[a] * s.r[a] * along[a]).sum() / total - mean[a] ** 2, min=0.0))
             for a in range(3)]
    mom = [(k[a] * kalong[a]).sum() / ktotal for a in range(3)]
    inside = (along[0] * (s.r[0] >= PAST)).sum() * s.dv
    return [float(v) for v in (total * s.dv, ev + et, ev, et, inside, *mean, *sigma, *mom)]


def _exact_steps(case, s):
    """The field after the pass, and for a relaxation the energy estimate of its last step."""
    k = _wavenumbers(s)
    k2 = (k[0] ** 2)[None, None, :] + (k[1] ** 2)[None, :, None] + (k[2] ** 2)[:, None, None]
    psi, energy = s.psi, None
    if case["precision"] == "c64":  # the run's own input
        psi = psi.to(torch.complex64).to(torch.complex128)
    if case["kind"] == "relax":
        half, kin = torch.exp(-0.5 * s.v * s.dt), torch.exp(-0.5 * k2 * s.dt)
        for _ in range(case["steps"]):
            psi = half * torch.fft.ifftn(kin * torch.fft.fftn(half * psi))
            n2 = psi.abs().square().sum() * s.dv
            psi = psi / torch.sqrt(n2)
            energy = -math.log(float(n2)) / (2.0 * s.dt)
        return psi, energy
    half = torch.polar(torch.ones_like(s.v), -0.5 * s.v * s.dt)
    kin = torch.polar(torch.ones_like(k2), -0.5 * k2 * s.dt)
    del k2
    after = half
    if case["absorb"]:
        m = [torch.from_numpy(a).cuda() for a in s.mask]
        after = half * (m[0][None, None, :] * m[1][None, :, None] * m[2][:, None, None])
    u = sum(c * r for c, r in zip(DRIVE["axis"], (s.x, s.y, s.z))) if case["kind"] == "driven" else None
    for i in range(case["steps"]):
        if u is not None:
            theta = [DRIVE["amplitude"] * math.cos(DRIVE["omega"] * t) * 0.5 * s.dt for t in (i * s.dt, (i + 1) * s.dt)]
            psi = psi * torch.exp(-1j * theta[0] * u)
        psi = torch.fft.ifftn(kin * torch.fft.fftn(half * psi)) * after
        if u is not None:
            psi = psi * torch.exp(-1j * theta[1] * u)
    return psi, energy


def exact(case, seed):
    psis, rows, density = [], [], None
    for s in _scenes(case, seed):
        psi, energy = _exact_steps(case, s)
        psis.append(psi)
        if case["kind"] == "relax":
            rows.append([energy])
        elif case["kind"] == "frame":
            w = psi.abs().square()
            density = w[case["nz"] // 2]
            rows.append([float(w.sum() * s.dv), float(w.max())])
        else:
            rows.append(_exact_row(s, psi))
    if case["kind"] == "batch":
        return dict(psi=psis, readings=np.array(rows))
    out = dict(psi=psis[0], readings=np.array(rows[0]))
    if density is not None:
        out["density"] = density
    return out
