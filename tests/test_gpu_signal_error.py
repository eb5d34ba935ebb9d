"""Error of the split-BF16 form where its accumulation, not the split, makes it:
like nodes, whose terms are equal, so that the sum of 512 nodes is 32 times that of
16 but for what the accumulators truncate."""
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
    stage to its main accumulator, 128; a wide one adds 6 and is folded after 21
    stages, 126 and then 66.  The truncation of a growing sum adds up to half an ulp
    an MMA over the mean of the sum, in proportion to the MMAs of a group: 0.82 times
    the narrow tile's on average, and 1.5 times if a wide tile collected 32 stages.
    The bound lies between."""
    def error(runs):
        few, many = _k(16, runs, cuda), _k(512, runs, cuda)
        return ((many / 32 - few).abs() / few.abs()).mean().item()
    wide, narrow = error(128), error(16)
    assert 0 < wide < 1.15 * narrow
