"""M of as many entries as rows that is not diagonal: rows of none, of a few and of
more entries than are taken one by one, several columns, columns of many entries."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from feelmri_b200 import ops, workloads as W
from feelmri_b200._motion import lower

pytestmark = pytest.mark.gpu


def _signal(M, V, precision, dev, seed=0, traj=None):
    n = M.shape[0]
    rng = np.random.default_rng(seed)
    traj = traj or W.cartesian(res=(6, 5, 4))
    real, cplx = (torch.float64, torch.complex128) if precision == "f64" else (torch.float32, torch.complex64)
    up = lambda a, d=real: torch.from_numpy(np.ascontiguousarray(a)).to(device=dev, dtype=d)  # noqa: E731
    inp = ops.SignalInputs(M=ops.SparseCSC(M.shape, up(M.indptr, torch.int32), up(M.indices, torch.int32), up(M.data)),
                           kx=up(traj.kx), ky=up(traj.ky), kz=up(traj.kz), t=up(traj.t),
                           r0=up(rng.uniform(-0.04, 0.04, (n, 3))), phi=up(W.off_resonance(n)),
                           T2=up(rng.uniform(50.0, 100.0, n)),
                           Mxy=up(rng.normal(size=(n, V)) + 1j * rng.normal(size=(n, V)), cplx))
    return inp, lower(None, n, dev)


def _matrix(kind, n):
    rng = np.random.default_rng(n)
    if kind == "permutation":
        at = rng.permutation(n), np.arange(n)
    elif kind == "one_row":
        at = np.full(n, n // 2), np.arange(n)
    elif kind == "one_column":
        at = rng.permutation(n), np.full(n, n // 3)
    elif kind == "rows_of_9":  # one more than is taken one by one
        at = np.repeat(np.arange(n // 9 + 1), 9)[:n] * 3 % n, rng.permutation(n)
    else:
        at = rng.integers(0, n, n) // 3, np.sort(rng.integers(0, n, n))
    order = np.lexsort((at[0], at[1]))  # by columns, duplicates kept
    indptr = np.searchsorted(at[1][order], np.arange(n + 1)).astype(np.int32)
    data = np.random.default_rng(1).uniform(1e-7, 3e-7, n)
    return sp.csc_matrix((data, at[0][order].astype(np.int32), indptr), shape=(n, n))


@pytest.mark.parametrize("precision,tol", [("f32", 1e-5), ("f64", 1e-12), ("bf16x3", 1e-4)])
@pytest.mark.parametrize("kind", ["permutation", "one_row", "one_column", "rows_of_9", "random"])
@pytest.mark.parametrize("n,V", [(1, 1), (2, 3), (257, 1), (1000, 9)])
def test_as_many_entries_as_rows(cuda, n, V, kind, precision, tol):
    """The same call on the product formed beforehand in 64 bits, with a unit matrix."""
    M = _matrix(kind, n)
    inp, motion = _signal(M, V, precision, cuda)
    K = ops.signal(inp, motion, precision)
    MM = torch.from_numpy(M.astype(np.float64) @ inp.Mxy.cpu().numpy().astype(np.complex128) * 1e7).to(cuda)
    inp.Mxy = MM.to(inp.Mxy.dtype).contiguous()
    inp.M = ops.SparseCSC((n, n), torch.arange(n + 1, dtype=torch.int32, device=cuda),
                          torch.arange(n, dtype=torch.int32, device=cuda), torch.ones_like(inp.M.data))
    ref = ops.signal(inp, motion, precision).to(torch.complex128) * 1e-7
    assert (torch.linalg.norm(K - ref) / torch.linalg.norm(ref)).item() < tol


def test_permuted_matrix_costs_little(cuda):
    """200,000 rows: the product of a permuted M is spread over the GPU as that of a
    diagonal one is (on a single block of threads it took nine times the whole
    call)."""
    n = 200_000

    def best(M):
        inp, motion = _signal(M, 2, "bf16x3", cuda, traj=W.cartesian(res=(32, 32, 8)))
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ops.signal(inp, motion, "bf16x3")
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)
    diagonal = best(sp.identity(n, format="csc") * 1e-7)
    assert best(_matrix("permutation", n)) < 2.0 * diagonal
