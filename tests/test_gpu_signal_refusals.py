"""Signal calls that the device work refuses: the call raises, and what would be
read out of range is not read."""
import numpy as np
import pytest
import torch

from feelmri_b200 import ops, workloads as W
from feelmri_b200._lib import FeelMRIError
from feelmri_b200._motion import lower, table_motion

pytestmark = pytest.mark.gpu


def _inputs(n, V, traj, precision, dev, seed=0):
    rng = np.random.default_rng(seed)
    real, cplx = (torch.float64, torch.complex128) if precision == "f64" else (torch.float32, torch.complex64)
    up = lambda a, d=real: torch.from_numpy(np.ascontiguousarray(a)).to(device=dev, dtype=d)  # noqa: E731
    idx = torch.arange(n + 1, dtype=torch.int32, device=dev)
    return ops.SignalInputs(M=ops.SparseCSC((n, n), idx, idx[:n], up(rng.uniform(1e-7, 3e-7, n))), kx=up(traj.kx),
                            ky=up(traj.ky), kz=up(traj.kz), t=up(traj.t), r0=up(rng.uniform(-0.04, 0.04, (n, 3))),
                            phi=up(W.off_resonance(n)), T2=up(rng.uniform(50.0, 100.0, n)),
                            Mxy=up(rng.normal(size=(n, V)) + 1j * rng.normal(size=(n, V)), cplx))


@pytest.mark.parametrize("precision", ["f32", "f64", "bf16x3"])
@pytest.mark.parametrize("kind", ["slabs", "samples"])
@pytest.mark.parametrize("entries", [1, 5, 7])
def test_table_of_another_number_of_runs(cuda, kind, precision, entries):
    """Six runs.  The table is the front of a larger one, so that the entries after
    it are memory of this test's own; the output stays as it was, since no node or
    sample of the problem is worked on."""
    n, V = 300, 2
    traj = W.cartesian(res=(6, 5, 4)) if kind == "slabs" else W.radial3d(n_ro=6, n_spokes=20, kmax=300.0)
    inp = _inputs(n, V, traj, precision, cuda)
    whole = torch.full((8, n, 3), 1e-3, dtype=inp.r0.dtype, device=cuda)
    out = torch.full((*traj.kx.shape, V), 7.0, dtype=inp.Mxy.dtype, device=cuda)
    with pytest.raises(ValueError, match="distinct-time run"):
        ops.signal(inp, table_motion(whole[:entries]), precision, out=out)
    assert (out == 7.0).all()
    # the right number, and the same displacement as a shift of the nodes
    K = ops.signal(inp, table_motion(whole[:6]), precision)
    inp.r0 = inp.r0 + 1e-3
    ref = ops.signal(inp, lower(None, n, cuda), precision)
    assert (torch.linalg.norm(K - ref) / torch.linalg.norm(ref)).item() < 1e-4


def test_table_of_another_number_of_runs_in_a_batch(cuda):
    n, V = 300, 1
    traj = W.cartesian(res=(6, 5, 4))
    inp = _inputs(n, V, traj, "bf16x3", cuda)
    whole = torch.full((8, n, 3), 1e-3, dtype=torch.float32, device=cuda)
    outs = [torch.full((*traj.kx.shape, V), 7.0, dtype=torch.complex64, device=cuda) for _ in range(2)]
    with pytest.raises(ValueError, match="distinct-time run"):
        ops.signal_batch([(inp, table_motion(whole[:6]), outs[0]), (inp, table_motion(whole[:5]), outs[1])])
    alone = ops.signal_batch([(inp, table_motion(whole[:6]), None)])[0]
    assert torch.equal(outs[0], alone) and (outs[1] == 7.0).all()


@pytest.mark.parametrize("kind", ["runs", "slabs", "samples"])
@pytest.mark.parametrize("phi,refused", [(float("nan"), True), (float("inf"), True), (-2.0 ** 26, True),
                                         (2.0 ** 22, False), (0.0, False)])
def test_off_resonance_out_of_range(cuda, kind, phi, refused):
    """The split-BF16 form reduces phi t as it does k . r: beyond its range (here t up
    to 32 ms or more, so 2^31 rad) the call fails instead of returning a finite wrong
    signal; 2^22 rad / ms is within it."""
    n = 200
    traj = W.radial3d(n_ro=40, n_spokes=30, kmax=300.0) if kind == "samples" else W.cartesian(res=(40, 6, 5))
    inp = _inputs(n, 1, traj, "bf16x3", cuda)
    inp.t = inp.t + 30.0
    inp.phi[7] = phi
    pod = W.sinusoidal_pod(n, n_modes=2) if kind == "slabs" else None
    motion = lower(pod, n, cuda)
    if refused:
        with pytest.raises(FeelMRIError, match="off-resonance"):
            ops.signal(inp, motion, "bf16x3")
        with pytest.raises(FeelMRIError, match="off-resonance"):
            ops.signal_batch([(inp, motion, None)])
    else:
        assert torch.isfinite(torch.view_as_real(ops.signal(inp, motion, "bf16x3"))).all()
    if kind == "slabs":
        return  # (nodes that move have no finite place at no time, which is refused)
    # a sample without a time is its own run of no finite signal, not a refusal
    inp.phi[7] = 0.1
    inp.t[3, 2] = float("nan")
    K = torch.view_as_real(ops.signal(inp, motion, "bf16x3"))
    assert K[3, 2].isnan().all() and K[4].isfinite().all()
