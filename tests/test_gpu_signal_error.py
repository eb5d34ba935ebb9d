"""Error where accumulation makes it.  The split-BF16 form on like nodes, whose terms
are equal, so that the sum of 512 nodes is 32 times that of 16 but for what the
accumulators truncate; the unfactored FP64 form on a plain sum."""
import math

import numpy as np
import pytest
import torch

from feelmri_b200 import ops, workloads as W
from feelmri_b200._motion import lower

pytestmark = pytest.mark.gpu


def _k(n, runs, dev):
    """k-space of n nodes at one place, one node range, `runs` columns a tile."""
    traj = W.cartesian(res=(runs, 16, 8))
    up = lambda a: torch.as_tensor(a, dtype=torch.float32, device=dev).contiguous()  # noqa: E731
    idx = torch.arange(n + 1, dtype=torch.int32, device=dev)
    one = torch.ones(n, device=dev)
    inp = ops.SignalInputs(M=ops.SparseCSC((n, n), idx, idx[:n], one * 1.234567e-7), kx=up(traj.kx), ky=up(traj.ky),
                           kz=up(traj.kz), t=up(traj.t), r0=up([[0.0123, -0.0234, 0.0171]]).expand(n, 3).contiguous(),
                           phi=one * 0.05, T2=one * 70.0,
                           Mxy=torch.full((n, 1), 0.3 + 0.2j, dtype=torch.complex64, device=dev))
    return ops.signal_batch([(inp, lower(None, n, dev), None)], ops.Tuning(split_nodes=1 << 20))[0].to(torch.complex128)


def test_wide_tiles_truncate_no_more_than_narrow_ones(cuda):
    """Each MMA on an accumulator truncates it.  A narrow tile of 32 stages adds 4 a
    stage to its main accumulator, 128; a wide one adds 6 and is folded after 12
    stages, 72.  The truncation of a growing sum adds up to half an ulp an MMA over
    the mean of the sum, in proportion to the MMAs of a group: about half the narrow
    tile's, and 1.5 times if a wide tile collected 32 stages.  The bound lies
    between."""
    def error(runs):
        few, many = _k(16, runs, cuda), _k(512, runs, cuda)
        return ((many / 32 - few).abs() / few.abs()).mean().item()
    wide, narrow = error(128), error(16)
    assert 0 < wide < 1.15 * narrow


def test_fp64_sums_are_cut(cuda):
    """592 tiles are four for each SM, so the nodes are not split.  Nodes at one place
    and samples at k = 0 of motion forms (unfactored): the result is the plain sum of
    M Mxy.  Rounding of a sum of n positive terms is some u sqrt(n) / 3 of it (u =
    2^-53): 47 u for 20,000 in one sum, 3 u in sums of 512."""
    n, V = 20_000, 8
    rng = np.random.default_rng(3)
    traj = W.radial3d(n_ro=592, n_spokes=4)
    up = lambda a, d=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(device=cuda, dtype=d)  # noqa: E731
    idx = torch.arange(n + 1, dtype=torch.int32, device=cuda)
    cols = rng.uniform(0.5, 1.5, (n, V)) + 1j * rng.uniform(0.5, 1.5, (n, V))
    inp = ops.SignalInputs(M=ops.SparseCSC((n, n), idx, idx[:n], up(np.ones(n))), kx=up(0 * traj.kx),
                           ky=up(0 * traj.ky), kz=up(0 * traj.kz), t=up(traj.t), r0=up(np.zeros((n, 3))),
                           phi=up(np.zeros(n)), T2=up(np.full(n, np.inf)), Mxy=up(cols, torch.complex128))
    motion = lower(W.sinusoidal_pod(n, n_modes=1), n, cuda)
    K = ops.signal(inp, motion, "f64").cpu().numpy().reshape(-1, V)
    assert (K == K[0]).all()  # every sample sums alike
    exact = np.array([complex(math.fsum(c.real), math.fsum(c.imag)) for c in cols.T])
    rel = np.concatenate([(K[0] - exact).real / exact.real, (K[0] - exact).imag / exact.imag])
    assert np.sqrt((rel ** 2).mean()) < 15 * 2.0 ** -53


def test_split_errors_of_nodes_in_line_are_independent(cuda):
    """Nodes of a regular grid, all alike, nothing moving: a row factor of place alone
    is the same for the 24 nodes of a line, and so is the error of its split.  The
    residual of a split is up to 2^-18 of an element, so with independent errors a
    sample is off by about 2^-18 of the root of the sum of squares, 3.8e-6 w sqrt(N);
    with the errors of a line in step, where the lines' own sums are large (the runs
    at kx about 0), by sqrt(24) times that.  The bound is 2 x 2^-18."""
    m, w = 24, 1.234567e-3
    n = m ** 3
    axis = (np.arange(m) - (m - 1) / 2) * 0.0031
    r0 = np.stack(np.meshgrid(axis, axis, axis, indexing="ij"), -1).reshape(-1, 3)
    traj = W.cartesian(res=(40, 40, 8))

    def form(precision):
        real, cplx = (torch.float64, torch.complex128) if precision == "f64" else (torch.float32, torch.complex64)
        up = lambda a: torch.from_numpy(np.ascontiguousarray(np.float32(a))).to(device=cuda, dtype=real)  # noqa: E731
        idx = torch.arange(n + 1, dtype=torch.int32, device=cuda)
        inp = ops.SignalInputs(M=ops.SparseCSC((n, n), idx, idx[:n], up(np.full(n, w))), kx=up(traj.kx), ky=up(traj.ky),
                               kz=up(traj.kz), t=up(traj.t), r0=up(r0), phi=up(np.zeros(n)), T2=up(np.full(n, 70.0)),
                               Mxy=torch.ones((n, 1), dtype=cplx, device=cuda))
        return ops.signal(inp, lower(None, n, cuda), precision).cpu().numpy()[..., 0].astype(np.complex128)
    K, ref = form("bf16x3"), form("f64")
    kx = np.abs(traj.kx)
    line = kx <= 1.01 * kx.min()             # the runs whose lines sum up
    weak = np.abs(ref) < 0.02 * n * w        # (at a peak the accumulators' rounding counts)
    assert (line & weak).sum() > 200
    assert np.sqrt((np.abs(K - ref)[line & weak] ** 2).mean()) < 2 * 2.0 ** -18 * w * np.sqrt(n)
