"""Performance cases of the simulation hot path.

Each case is one call that a simulation makes, through the package's public
entry points, on device-resident inputs (the reconstruction works on host
arrays, as its callers do).  `listed()` names the cases that are tracked,
`draw(rng)` gives more of the same ranges, `prepare` makes a case's inputs,
`run` is one pass, `work` what the pass cannot do without and `exact` the same
outputs in 64 bits from plain torch / numpy.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from feelmri_b200 import Recon, ops
from feelmri_b200 import workloads as W
from feelmri_b200._motion import lower
from feelmri_b200.FiniteElements import FiniteElement, QuadratureRule
from feelmri_b200.motion import SplineMotion, SplineTerm
from feelmri_b200.serving import SERVING_TUNING

# the Signal's 2 pi is built from a float32-rounded pi (cpp/feelmri/MRI.h:13)
TWO_PI = 2.0 * float(np.float32(np.pi))
PERIOD = 800.0   # ms, cardiac cycle of the mode motion
FRAMES = 40      # spline knots per cycle

# Body sizes in metres, as the phantoms of the benchmark use them.
TUBE_RADIUS, TUBE_LENGTH = 0.012, 0.1
AXES = (0.06, 0.05, 0.04)


def listed():
    return [
        # one repetition of a spoiled gradient echo on a small phantom, final
        # state only: the smallest call, launched once per block
        dict(name="bloch_block_small", kind="bloch", nodes=5003, block="gre", tr=5.0, motion="none", modes=0,
             history=False),
        # the drop-in solve_mri's history form on the 200k-node flow phantom
        # (one velocity-encoded block, nodes moving with the flow)
        dict(name="bloch_history_flow", kind="bloch", nodes=200740, block="flow", tr=5.0, motion="flow", modes=1,
             history=True),
        # BlochSolver's block sequence: imaging blocks with empty spacing
        # blocks up to TR 40 ms, on nodes that move with four cardiac modes
        dict(name="bloch_sequence", kind="sequence", nodes=100003, imaging=24, stored=4, spacing=40.0, motion="modes",
             modes=4),
        # the plain configuration's readout: 20k nodes, 64 x 64, one coil, FP64
        dict(name="signal_f64_plane", kind="signal", precision="f64", traj="cartesian", nodes=20011, ro=64, lines=64,
             kz=1, fov=0.1, columns=1, motion="none", modes=0),
        # the drop-in default (float32 arrays) on a flow phantom with four
        # velocity encodings, a reduced 3-D Cartesian matrix
        dict(name="signal_f32_flow", kind="signal", precision="f32", traj="cartesian", nodes=50021, ro=48, lines=48,
             kz=16, fov=0.1, columns=4, motion="flow", modes=1),
        # float32 arrays on a non-Cartesian readout with eight coils
        dict(name="signal_f32_radial", kind="signal", precision="f32", traj="radial", nodes=20011, ro=128, lines=255,
             kz=1, fov=0.1, columns=8, motion="none", modes=0),
        # the smallest tensor-core Signal: one frame of a small served request
        dict(name="signal_bf16x3_small", kind="signal", precision="bf16x3", traj="cartesian", nodes=3083, ro=16,
             lines=16, kz=8, fov=0.1, columns=1, motion="none", modes=0),
        # phase-contrast flow at full size: 200k nodes, 96 x 96 x 32, 4 encodings
        dict(name="signal_bf16x3_flow", kind="signal", precision="bf16x3", traj="cartesian", nodes=200740, ro=96,
             lines=96, kz=32, fov=0.1, columns=4, motion="flow", modes=1),
        # the precision configuration at reduced size: 3-D radial, eight coils,
        # ten cardiac modes
        dict(name="signal_bf16x3_radial", kind="signal", precision="bf16x3", traj="radial", nodes=50021, ro=128,
             lines=512, kz=1, fov=0.1, columns=8, motion="modes", modes=10),
        # the batched configuration: phantoms of uneven size, Cartesian grids
        # and stacks of spirals, in one persistent launch
        dict(name="signal_batch_uneven", kind="batch", phantoms=16, nodes_min=5000, nodes_max=150000,
             samples_min=4000, samples_max=120000, layout=4),
        # image reconstruction: the adjoint from radial k-space of four coils
        # onto a voxel grid, host arrays in and out
        dict(name="recon_adjoint_radial", kind="recon", ro=128, spokes=510, columns=4, nx=64, ny=64, nz=24, fov=0.2),
        # set-up of a phantom: the consistent P1 mass matrix of a tetrahedral mesh
        dict(name="mass_assemble_f64", kind="mass", precision="f64", nodes=60000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges; no drawn case costs more than
    the largest listed one (signal_bf16x3_flow)."""
    kind = rng.choice(["bloch", "bloch", "sequence", "f64", "f32", "f32", "bf16x3", "bf16x3", "bf16x3", "batch", "recon",
                       "mass"])
    if kind == "bloch":
        motion = rng.choice(["none", "flow", "modes"])
        history = rng.random() < 0.5
        return dict(kind="bloch", nodes=_log(rng, 3000, 200000 if history else 400000),
                    block=rng.choice(["gre", "flow", "spamm"]), tr=rng.choice([4.0, 5.0, 8.0]), motion=motion,
                    modes={"none": 0, "flow": 1, "modes": rng.randint(2, 12)}[motion], history=history)
    if kind == "sequence":
        motion = rng.choice(["none", "flow", "modes"])
        imaging = rng.randint(4, 40)
        return dict(kind="sequence", nodes=_log(rng, 5000, 150000), imaging=imaging, stored=rng.randint(1, 4),
                    spacing=rng.choice([10.0, 25.0, 40.0]), motion=motion,
                    modes={"none": 0, "flow": 1, "modes": rng.randint(2, 10)}[motion])
    if kind == "batch":
        return dict(kind="batch", phantoms=rng.randint(4, 20), nodes_min=4000, nodes_max=_log(rng, 20000, 150000),
                    samples_min=2000, samples_max=_log(rng, 10000, 120000), layout=rng.randint(5, 1 << 20))
    if kind == "recon":
        return dict(kind="recon", ro=rng.randint(48, 160), spokes=rng.randint(100, 800), columns=rng.randint(1, 8),
                    nx=rng.randint(24, 80), ny=rng.randint(24, 80), nz=rng.randint(8, 32),
                    fov=rng.choice([0.15, 0.2, 0.25]))
    if kind == "mass":
        return dict(kind="mass", precision=rng.choice(["f32", "f64"]), nodes=_log(rng, 5000, 150000))
    motion = rng.choice(["none", "none", "flow", "modes"])
    traj = rng.choice(["cartesian", "cartesian", "spiral", "radial"])
    nodes, ro, lines, kz, columns = {
        "f64": (_log(rng, 5000, 40000), rng.randint(24, 80), rng.randint(24, 80), rng.choice([1, 1, 4]),
                rng.randint(1, 4)),
        "f32": (_log(rng, 4000, 80000), rng.randint(24, 64), rng.randint(24, 64), rng.choice([1, 4, 9, 16]),
                rng.randint(1, 8)),
        "bf16x3": (_log(rng, 3000, 200000), rng.randint(16, 96), rng.randint(16, 96), rng.choice([1, 8, 12, 16, 31]),
                   rng.randint(1, 8)),
    }[kind]
    if traj == "spiral":
        ro, lines = ro * rng.randint(4, 10), max(2, lines // 8)
    elif traj == "radial":
        lines, kz = lines * max(kz // 2, 1) + rng.randint(0, 3), 1
    # node-samples times columns, bounded by what the largest listed case takes:
    # one sin/cos per node-sample outside the factored slabs
    dense = traj == "radial" or kz == 1
    most = {"f64": 6e8, "f32": 3e9 / (1 + columns / 8), "bf16x3": 3e9 if dense else min(3e10, 2.3e11 / columns)}[kind]
    nodes = max(1000, min(nodes, int(most / (ro * lines * kz))))
    return dict(kind="signal", precision=kind, traj=traj, nodes=nodes, ro=ro, lines=lines, kz=kz,
                fov=rng.choice([0.1, 0.1, 0.15, 0.256, 0.3]), columns=columns, motion=motion,
                modes={"none": 0, "flow": 1, "modes": rng.randint(2, 12)}[motion])


# ------------------------------------------------------------------- inputs --

def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _nodes(n, body, rng):
    """n points spread evenly over a tube (along z) or an ellipsoid."""
    u = rng.random((n, 3))
    if body == "tube":
        rho, a = TUBE_RADIUS * np.sqrt(u[:, 0]), 2 * np.pi * u[:, 1]
        p = np.stack([rho * np.cos(a), rho * np.sin(a), TUBE_LENGTH * (u[:, 2] - 0.5)], axis=1)
    else:
        rho, a, c = np.cbrt(u[:, 0]), 2 * np.pi * u[:, 1], 2 * u[:, 2] - 1
        s = np.sqrt(1 - c * c)
        p = np.stack([rho * s * np.cos(a), rho * s * np.sin(a), rho * c], axis=1) * np.asarray(AXES)
    return p.astype(np.float32)


def _hermite(values, slopes, h):
    """Power-basis coefficients (4, n - 1, r), highest power first, of the
    cubic Hermite interpolant with knot spacing h."""
    y0, y1, d0, d1 = values[:-1], values[1:], slopes[:-1], slopes[1:]
    return np.stack([(2 * (y0 - y1) + h * (d0 + d1)) / h ** 3, (3 * (y1 - y0) - h * (2 * d0 + d1)) / h ** 2, d0, y0])


def _motion(case, pos, rng):
    """The case's motion and (modes, coefficients, knots, velocity) for exact()."""
    n = pos.shape[0]
    if case["motion"] == "none":
        return None, None
    if case["motion"] == "flow":
        # Poiseuille flow along z, peak 1 m/s, as one velocity mode
        rho2 = pos[:, 0].astype(np.float64) ** 2 + pos[:, 1].astype(np.float64) ** 2
        modes = np.zeros((n, 3, 1), np.float32)
        modes[:, 2, 0] = np.clip(1 - rho2 / TUBE_RADIUS ** 2, 0, None) / 1000.0
        knots = np.linspace(0.0, 1000.0, 20)
        coeffs = np.zeros((4, 19, 1))
        coeffs[3] = 1.0
        period = 1000.0
    else:
        # cardiac modes of about a millimetre with sinusoidal weights
        r = case["modes"]
        modes = rng.normal(0.0, 1e-3 / math.sqrt(r), (n, 3, r)).astype(np.float32)
        knots = np.linspace(0.0, PERIOD, FRAMES)
        arg = 2 * np.pi * knots[:, None] / PERIOD + rng.uniform(0, 2 * np.pi, r)[None, :]
        coeffs = _hermite(np.sin(arg), 2 * np.pi / PERIOD * np.cos(arg), knots[1])
        period = PERIOD
    flow = case["motion"] == "flow"
    term = SplineTerm("velocity_modes" if flow else "modes", coeffs, knots, modes=modes, period=period)
    return SplineMotion([term]), (modes, coeffs, knots, period, flow)


def _displacement(exact_motion, t, shift, dev):
    """Displacement (N, 3) float64 at time t of a motion from _motion."""
    modes, coeffs, knots, period, velocity = exact_motion
    tau = t + shift
    tau -= period * math.floor(tau / period)
    i = min(max(int(np.searchsorted(knots, tau, side="right")) - 1, 0), len(knots) - 2)
    h = tau - knots[i]
    w = ((coeffs[0, i] * h + coeffs[1, i]) * h + coeffs[2, i]) * h + coeffs[3, i]
    if velocity:
        w = w * t
    return _f64(modes, dev) @ torch.from_numpy(np.ascontiguousarray(w)).to(dev)


def _f64(a, dev):
    if isinstance(a, torch.Tensor):
        return a.to(device=dev, dtype=torch.complex128 if a.is_complex() else torch.float64)
    a = np.asarray(a)
    return torch.from_numpy(np.ascontiguousarray(a.astype(np.complex128 if np.iscomplexobj(a) else np.float64))).to(dev)


def _up(a, dtype, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(device=dev, dtype=dtype)


def _block(case):
    if case["block"] == "gre":
        return W.hard_pulse_block(0.0, 15.0, case["tr"])
    if case["block"] == "spamm":
        return W.spamm_block(0.0, tail=case["tr"])
    return W.pc_imaging_block(0.0, (0, 0, 1), tr=case["tr"])


def _sequence_blocks(case):
    """Imaging blocks, each followed by an empty spacing block in 1 ms steps."""
    blocks, t = [], 0.0
    for i in range(case["imaging"]):
        b = W.pc_imaging_block(t, (1, 0, 0))
        b.store_magnetization = i >= case["imaging"] - case["stored"]
        dur = float(b.times[-1] - b.times[0])
        g = W.hard_pulse_block(t + dur, 0.0, case["spacing"] - dur, dt=1.0)
        g.empty = True
        blocks += [b, g]
        t += case["spacing"]
    return blocks


def _bloch_host(case, seed):
    rng = np.random.default_rng([11, seed])
    n = case["nodes"]
    pos = _nodes(n, "tube" if case["motion"] == "flow" else "ellipsoid", rng)
    T1 = rng.uniform(800.0, 1200.0, n).astype(np.float32)
    T2 = rng.uniform(50.0, 100.0, n).astype(np.float32)
    # a static field error of about 20 Hz, as mT
    dB = (2 * np.pi * rng.normal(0.0, 20.0, n) / 1000.0 / W.GAMMA).astype(np.float32)
    mz = rng.uniform(0.6, 1.0, n).astype(np.float32)
    pod, ex = _motion(case, pos, rng)
    return dict(pos=pos, T1=T1, T2=T2, dB=dB, mz=mz, pod=pod, ex=ex)


def _trajectory(case):
    fov, ro, lines, kz = case["fov"], case["ro"], case["lines"], case["kz"]
    if case["traj"] == "cartesian":
        return W.cartesian(res=(ro, lines, kz), fov=(fov, fov, fov))
    if case["traj"] == "spiral":
        return W.spiral_stack(n_ro=ro, n_interleaves=lines, n_kz=kz, fov=fov)
    return W.radial3d(n_ro=ro, n_spokes=lines, kmax=ro / (2 * fov))


def _signal_host(case, seed):
    """Node and k-space arrays of one Signal call: lumped mass weights of an
    even mesh, magnetisation after a 15 degree pulse seen through coils, or
    four velocity encodings of the flow."""
    rng = np.random.default_rng([12, seed])
    n, V = case["nodes"], case["columns"]
    pos = _nodes(n, "tube" if case["motion"] == "flow" else "ellipsoid", rng)
    T2 = rng.uniform(50.0, 100.0, n).astype(np.float32)
    phi = (2 * np.pi * rng.normal(0.0, 20.0, n) / 1000.0).astype(np.float32)
    mass = (rng.uniform(0.5, 1.5, n) * 1e-4 / n).astype(np.float32)
    m = math.sin(math.radians(15.0)) * rng.uniform(0.8, 1.0, n)
    if case["motion"] == "flow":
        # velocity phases of the encodings (one venc of 1.5 m/s is pi)
        speed = 1 - (pos[:, 0].astype(np.float64) ** 2 + pos[:, 1].astype(np.float64) ** 2) / TUBE_RADIUS ** 2
        cols = np.stack([m * np.exp(1j * np.pi * speed / 1.5 * (v % 4 == 3)) * np.exp(0.1j * v) for v in range(V)],
                        axis=1).astype(np.complex64)
    else:
        cols = (m[:, None] * W.coil_maps(pos, V, seed=seed)).astype(np.complex64)
    pod, ex = _motion(case, pos, rng)
    return dict(pos=pos, T2=T2, phi=phi, mass=mass, cols=cols, traj=_trajectory(case), pod=pod, ex=ex)


def _batch_cases(case):
    """The phantoms of a batch: node and sample counts log-uniform, Cartesian
    grids and stacks of spirals in turn, one or two coils."""
    rng = np.random.default_rng([13, case["layout"]])
    out = []
    for i in range(case["phantoms"]):
        n = int(np.exp(rng.uniform(np.log(case["nodes_min"]), np.log(case["nodes_max"]))))
        s = np.exp(rng.uniform(np.log(case["samples_min"]), np.log(case["samples_max"])))
        kz = int(rng.choice([8, 16, 32]))
        if i % 2 == 0:
            ro = lines = max(4, int(round(np.sqrt(s / kz))))
        else:
            lines = int(rng.choice([8, 16, 32]))
            ro = max(16, int(round(s / (lines * kz))))
        out.append(dict(traj="cartesian" if i % 2 == 0 else "spiral", nodes=n, ro=ro, lines=lines, kz=kz, fov=0.1,
                        columns=int(rng.integers(1, 3)), motion="none", modes=0))
    return out


def _signal_state(h, precision):
    dev = _device()
    real, cplx = (torch.float64, torch.complex128) if precision == "f64" else (torch.float32, torch.complex64)
    n, t = h["pos"].shape[0], h["traj"]
    idx = torch.arange(n + 1, dtype=torch.int32, device=dev)
    inp = ops.SignalInputs(M=ops.SparseCSC((n, n), idx, idx[:n], _up(h["mass"], real, dev)), kx=_up(t.kx, real, dev),
                           ky=_up(t.ky, real, dev), kz=_up(t.kz, real, dev), t=_up(t.t, real, dev),
                           r0=_up(h["pos"], real, dev), phi=_up(h["phi"], real, dev), T2=_up(h["T2"], real, dev),
                           Mxy=_up(h["cols"], cplx, dev))
    return inp, lower(h["pod"], n, dev)


def _mesh(case, seed):
    """A cylinder's tetrahedra, the nodes jittered by a tenth of the spacing."""
    rng = np.random.default_rng([14, seed])
    mesh = W.cylinder(case["nodes"])
    h = (np.pi * 0.04 ** 2 * 0.08 / mesh.n_nodes) ** (1 / 3)
    nodes = mesh.nodes + rng.uniform(-0.1 * h, 0.1 * h, mesh.nodes.shape)
    return mesh.elems, nodes.astype(np.float64 if case["precision"] == "f64" else np.float32)


def _recon_host(case, seed):
    rng = np.random.default_rng([15, seed])
    t = W.radial3d(n_ro=case["ro"], n_spokes=case["spokes"], kmax=case["nx"] / (2 * case["fov"]))
    k = np.stack([t.kx, t.ky, t.kz]).reshape(3, -1)
    rho = np.sqrt((k.astype(np.float64) ** 2).sum(0)) * case["fov"]
    # k-space of a blurred object: large near the centre, falling outwards, and noise
    K = (np.exp(-0.5 * (rho / 4.0) ** 2)[:, None] * np.exp(2j * np.pi * rng.random((1, case["columns"]))) +
         0.01 * (rng.normal(size=(rho.size, case["columns"])) + 1j * rng.normal(size=(rho.size, case["columns"]))))
    dcw = (rho ** 2 / (rho ** 2).mean() + 1e-3).astype(np.float32)
    return K.astype(np.complex64), t, dcw


def prepare(case, seed):
    dev = _device()
    kind = case["kind"]
    if kind == "bloch":
        h, b = _bloch_host(case, seed), _block(case)
        inp = ops.BlochInputs(r0=_up(h["pos"], torch.float32, dev), T1=_up(h["T1"], torch.float32, dev),
                              T2=_up(h["T2"], torch.float32, dev), delta_B=_up(h["dB"], torch.float32, dev), M0=1.0,
                              gamma=W.GAMMA, rf=_up(b.rf, torch.complex64, dev), G=_up(b.G, torch.float32, dev),
                              dt=_up(b.dt, torch.float32, dev),
                              Mxy0=torch.zeros(case["nodes"], dtype=torch.complex64, device=dev),
                              Mz0=_up(h["mz"], torch.float32, dev))
        return dict(kind=kind, inp=inp, motion=lower(h["pod"], case["nodes"], dev), history=case["history"])
    if kind == "sequence":
        h, blocks, n = _bloch_host(case, seed), _sequence_blocks(case), case["nodes"]
        table, stored = [], 0
        for b in blocks:
            shifts = ((b.t0, 1),) if h["pod"] is not None else ()
            table.append(ops.SequenceBlock(n_time=b.times.size, empty=b.empty,
                                           store=stored if b.store_magnetization else -1, timeshifts=shifts))
            stored += int(b.store_magnetization)
        new = lambda *s, dtype: torch.empty(s, dtype=dtype, device=dev)  # noqa: E731
        return dict(kind=kind, r0=_up(h["pos"], torch.float32, dev), T1=_up(h["T1"], torch.float32, dev),
                    T2=_up(h["T2"], torch.float32, dev), dB=_up(h["dB"], torch.float32, dev), blocks=table,
                    rf=_up(np.concatenate([b.rf for b in blocks]), torch.complex64, dev),
                    G=_up(np.concatenate([b.G for b in blocks]), torch.float32, dev),
                    dt=_up(np.concatenate([b.dt for b in blocks]), torch.float32, dev),
                    m0=torch.zeros(n, dtype=torch.complex64, device=dev), z0=_up(h["mz"], torch.float32, dev),
                    motion=lower(h["pod"], n, dev), m=new(stored, n, dtype=torch.complex64),
                    z=new(stored, n, dtype=torch.float32), mc=new(n, dtype=torch.complex64),
                    zc=new(n, dtype=torch.float32))
    if kind == "signal":
        inp, motion = _signal_state(_signal_host(case, seed), case["precision"])
        return dict(kind=kind, inp=inp, motion=motion, precision=case["precision"])
    if kind == "batch":
        problems = []
        for i, c in enumerate(_batch_cases(case)):
            inp, motion = _signal_state(_signal_host(c, 1000 * seed + i), "bf16x3")
            problems.append((inp, motion, None))
        return dict(kind=kind, problems=problems)
    if kind == "recon":
        K, t, dcw = _recon_host(case, seed)
        return dict(kind=kind, K=K, traj=t, dcw=dcw, shape=(case["nx"], case["ny"], case["nz"]),
                    fov=(case["fov"],) * 3)
    elems, nodes = _mesh(case, seed)
    real = torch.float64 if case["precision"] == "f64" else torch.float32
    fe, qr = FiniteElement(dtype=np.float64), QuadratureRule(order=2, dtype=np.float64)
    tab = np.stack([fe.tabulate(1, qr.points[q:q + 1])[:, 0, :, 0] for q in range(len(qr.weights))])
    return dict(kind=kind, elems=_up(elems, torch.int32, dev), nodes=_up(nodes, real, dev),
                qw=_up(qr.weights, real, dev), tab=_up(tab, real, dev))


def run(state):
    s = state
    if s["kind"] == "bloch":
        return list(ops.bloch_solve(s["inp"], s["motion"], history=s["history"]))
    if s["kind"] == "sequence":
        ops.bloch_sequence(s["r0"], s["T1"], s["T2"], s["dB"], 1.0, W.GAMMA, s["blocks"], s["rf"], s["G"], s["dt"],
                           s["m0"], s["z0"], s["motion"], s["m"], s["z"], Mxy_carry=s["mc"], Mz_carry=s["zc"])
        return [s["m"], s["z"], s["mc"], s["zc"]]
    if s["kind"] == "signal":
        return ops.signal(s["inp"], s["motion"], s["precision"])
    if s["kind"] == "batch":
        return ops.signal_batch(s["problems"], SERVING_TUNING)
    if s["kind"] == "recon":
        t = s["traj"]
        return Recon.nudft_adjoint(s["K"], t.kx, t.ky, t.kz, s["shape"], s["fov"], dcw=s["dcw"])
    return list(ops.mass_assemble(s["elems"], s["nodes"], s["qw"], s["tab"]))


# --------------------------------------------------------------------- work --

def _signal_work(c, real=4):
    n, s, v = c["nodes"], c["ro"] * c["lines"] * c["kz"], c["columns"]
    return dict(bytes=n * (3 + 2 + 1 + 2 * v + 3 * c["modes"]) * real + s * (4 + 2 * v) * real, flops=8.0 * n * s * v)


def work(case):
    kind = case["kind"]
    if kind in ("bloch", "sequence"):
        n = case["nodes"]
        blocks = [_block(case)] if kind == "bloch" else _sequence_blocks(case)
        steps = sum(b.times.size - 1 for b in blocks)
        out = (steps + 1 if case["history"] else 1) if kind == "bloch" else case["stored"] + 1
        # the rotation and relaxation of a step: 20 multiply-adds
        return dict(bytes=n * (12 + 12 + 12 + 12 * case["modes"] + 12 * out), flops=40.0 * n * steps)
    if kind == "signal":
        return _signal_work(case, 8 if case["precision"] == "f64" else 4)
    if kind == "batch":
        parts = [_signal_work(c) for c in _batch_cases(case)]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    if kind == "recon":
        s, n, v = case["ro"] * case["spokes"], case["nx"] * case["ny"] * case["nz"], case["columns"]
        return dict(bytes=s * (16 + 8 * v) + 8 * n * v, flops=8.0 * n * s * v)
    n, real = case["nodes"], 8 if case["precision"] == "f64" else 4
    e, nnz = 5.5 * n, 15.0 * n
    return dict(bytes=e * 16 + n * 3 * real + nnz * (4 + real) + 4 * n, flops=60.0 * e)


# -------------------------------------------------------------------- exact --

def _bloch_steps(h, blocks, dev, history=False):
    """The rotation and relaxation of every step in 64 bits."""
    pos, dB = _f64(h["pos"], dev), _f64(h["dB"], dev)
    T1, T2 = _f64(h["T1"], dev), _f64(h["T2"], dev)
    gamma = float(np.float32(W.GAMMA))
    m, z = torch.zeros(pos.shape[0], dtype=torch.complex128, device=dev), _f64(h["mz"], dev)
    out = []
    if history:
        out.append((m, z))
    for b in blocks:
        rf, G, dt = b.rf.astype(np.complex128), b.G.astype(np.float64), b.dt.astype(np.float32).astype(np.float64)
        t = 0.0
        for i in range(1, b.times.size):
            t += dt[i]
            r = pos if h["ex"] is None else pos + _displacement(h["ex"], t, b.t0 if len(blocks) > 1 else 0.0, dev)
            Bz = r @ torch.from_numpy(G[i]).to(dev) + dB
            B = torch.clamp(torch.sqrt(Bz * Bz + abs(rf[i]) ** 2), min=1e-12)
            half = -0.5 * gamma * dt[i] * B
            c, s = torch.cos(half), torch.sin(half)
            al = torch.complex(c, -Bz / B * s)
            be = -1j * complex(rf[i]) * (s / B)
            ca = al.conj()
            m, z = (2 * ca * be * z + ca * ca * m - be * be * m.conj(),
                    (al.abs() ** 2 - be.abs() ** 2) * z - 2 * (al * be * m.conj()).real)
            e1 = torch.exp(-dt[i] / T1)
            m, z = m * torch.exp(-dt[i] / T2), z * e1 + (1 - e1)
            if history:
                out.append((m, z))
        if len(blocks) > 1:
            if b.store_magnetization:
                out.append((m, z))
            if not b.empty:
                m = 0 * m
    return out, m, z


def _phases(k, r, out_dtype=torch.complex128):
    """exp(-i 2 pi k . r), (len(k), len(r))."""
    ph = (k @ r.T) * TWO_PI
    return torch.complex(torch.cos(ph), -torch.sin(ph)).to(out_dtype)


def _signal_exact(c, h, dev, two_pi=TWO_PI):
    """The sum over the nodes in 64 bits, one readout index (one sample time)
    at a time; a (line, kz) slab with k = kp + kq as a product of two factors."""
    t = h["traj"]
    pos, phi, T2 = _f64(h["pos"], dev), _f64(h["phi"], dev), _f64(h["T2"], dev)
    MM = _f64(h["mass"], dev)[:, None] * _f64(h["cols"], dev)
    k = torch.stack([_f64(a, dev) for a in (t.kx, t.ky, t.kz)], dim=-1)  # (ro, lines, kz, 3)
    times = np.asarray(t.t, np.float64)[:, 0, 0]
    n, V = MM.shape
    ro, lines, kz = t.shape
    out = torch.zeros((ro, lines, kz, V), dtype=torch.complex128, device=dev)
    step = max(1024, (1 << 25) // max(lines, kz * V))
    for i in range(ro):
        r = pos if h["ex"] is None else pos + _displacement(h["ex"], float(times[i]), 0.0, dev)
        Wt = MM * torch.polar(torch.exp(-times[i] / T2), phi * times[i])[:, None]
        for a in range(0, n, step):
            A = _phases(k[i, :, 0], r[a:a + step])
            if kz == 1:
                out[i, :, 0] += A @ Wt[a:a + step]
                continue
            B = _phases(k[i, 0] - k[i, 0, :1], r[a:a + step])  # (kz, n)
            BW = (B.T[:, :, None] * Wt[a:a + step, None, :]).reshape(-1, kz * V)
            out[i] += (A @ BW).reshape(lines, kz, V)
    return out


def exact(case, seed):
    dev = _device()
    kind = case["kind"]
    if kind == "bloch":
        out, m, z = _bloch_steps(_bloch_host(case, seed), [_block(case)], dev, history=case["history"])
        if case["history"]:
            return [torch.stack([o[0] for o in out]), torch.stack([o[1] for o in out])]
        return [m, z]
    if kind == "sequence":
        out, m, z = _bloch_steps(_bloch_host(case, seed), _sequence_blocks(case), dev)
        return [torch.stack([o[0] for o in out]), torch.stack([o[1] for o in out]), m, z]
    if kind == "signal":
        return _signal_exact(case, _signal_host(case, seed), dev)
    if kind == "batch":
        return [_signal_exact(c, _signal_host(c, 1000 * seed + i), dev) for i, c in enumerate(_batch_cases(case))]
    if kind == "recon":
        K, t, dcw = _recon_host(case, seed)
        ax = [(np.arange(n) - n // 2) * (case["fov"] / n) for n in (case["nx"], case["ny"], case["nz"])]
        ax = [_f64(a.astype(np.float32), dev) for a in ax]
        Wk = _f64(K, dev) * _f64(dcw, dev)[:, None]
        e = [_phases(-a[:, None], _f64(g.reshape(-1), dev)[:, None]) for a, g in zip(ax, (t.kx, t.ky, t.kz))]
        S, V = Wk.shape
        out = torch.zeros((case["nx"], case["ny"], case["nz"] * V), dtype=torch.complex128, device=dev)
        for a in range(0, S, 1 << 14):
            z = (e[2][:, a:a + (1 << 14)].T[:, :, None] * Wk[a:a + (1 << 14), None, :]).reshape(-1, case["nz"] * V)
            for i in range(case["nx"]):
                out[i] += (e[1][:, a:a + (1 << 14)] * e[0][i, a:a + (1 << 14)]) @ z
        return out.reshape(case["nx"], case["ny"], case["nz"], V)
    # P1 on a tetrahedron: |det| / 6 times (1 + delta_ij) / 20
    elems, nodes = _mesh(case, seed)
    el, X = torch.from_numpy(elems.astype(np.int64)).to(dev), _f64(nodes, dev)
    vol = torch.linalg.det(X[el[:, 1:]] - X[el[:, :1]]).abs() / 6
    local = vol[:, None, None] * (torch.ones(4, 4, dtype=torch.float64, device=dev) +
                                  torch.eye(4, dtype=torch.float64, device=dev)) / 20
    n = nodes.shape[0]
    key = (el[:, None, :] * n + el[:, :, None]).reshape(-1)  # column, then row
    uniq, inv = torch.unique(key, return_inverse=True)
    data = torch.zeros(uniq.numel(), dtype=torch.float64, device=dev).index_add_(0, inv, local.reshape(-1))
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    indptr[1:] = torch.cumsum(torch.bincount(uniq // n, minlength=n), 0)
    return [indptr, uniq % n, data]
