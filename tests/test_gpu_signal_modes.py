"""POD modes that the tensor-core Signal reads from global memory, in each width
that their rows' alignment allows: the same bits whatever the address, and the
FP64 form's result."""
import numpy as np
import pytest
import torch

from feelmri_b200 import ops, workloads as W
from feelmri_b200._motion import lower

pytestmark = pytest.mark.gpu


def _inputs(n, V, traj, dev, real):
    rng = np.random.default_rng(n)
    cplx = torch.complex128 if real == torch.float64 else torch.complex64
    up = lambda a, d=real: torch.from_numpy(np.ascontiguousarray(np.float32(a) if d != cplx else a)).to(dev, d)  # noqa: E731
    idx = torch.arange(n + 1, dtype=torch.int32, device=dev)
    return ops.SignalInputs(M=ops.SparseCSC((n, n), idx, idx[:n], up(rng.uniform(1e-7, 3e-7, n))), kx=up(traj.kx),
                            ky=up(traj.ky), kz=up(traj.kz), t=up(traj.t), r0=up(rng.uniform(-0.04, 0.04, (n, 3))),
                            phi=up(W.off_resonance(n)), T2=up(rng.uniform(50.0, 100.0, n)),
                            Mxy=up(rng.normal(size=(n, V)) + 1j * rng.normal(size=(n, V)), cplx))


@pytest.mark.parametrize("modes", [1, 11, 14, 20, 33, 64])
@pytest.mark.parametrize("kind", ["slabs", "samples"])
def test_modes_read_in_any_width(cuda, kind, modes):
    n, V = 700, 2
    traj = W.cartesian(res=(4, 9, 5)) if kind == "slabs" else W.radial3d(n_ro=4, n_spokes=40, kmax=300.0)
    pod = W.sinusoidal_pod(n, n_modes=modes, amp=1e-3, period=50.0, n_frames=8)
    rows = torch.from_numpy(np.ascontiguousarray(pod.terms[0].modes, np.float32).reshape(-1))
    inp = _inputs(n, V, traj, cuda, torch.float32)
    out = []
    for shift in (0, 1, 2):  # floats: rows at 16, 4 and 8 bytes
        buf = torch.empty(rows.numel() + 4, dtype=torch.float32, device=cuda)[shift:shift + rows.numel()]
        buf.copy_(rows)
        motion = lower(pod, n, cuda)
        motion.struct.terms[0].modes = buf.data_ptr()
        motion.keep.append(buf)
        out.append(ops.signal(inp, motion, "bf16x3"))
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
    ref = ops.signal(_inputs(n, V, traj, cuda, torch.float64), lower(pod, n, cuda), "f64")
    assert (torch.linalg.norm(out[0] - ref) / torch.linalg.norm(ref)).item() < 1e-4
