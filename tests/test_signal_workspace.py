"""Device memory that a Signal call asks for, from the size queries (no GPU): the
partial sums of its node splits stay within what the calls state."""
import ctypes as C

import pytest

from feelmri_b200 import _lib as L
from feelmri_b200.ops import PRECISIONS

MB = 1 << 20


def _args(n, V, grid):
    a = L.SignalArgs()
    a.n_nodes = a.m_rows = a.m_cols = a.m_nnz = n
    a.n_vencs = V
    a.n_ro, a.n_lines, a.n_kz = grid
    for name in ("kx", "ky", "kz", "t", "r0", "phi", "T2", "Mxy", "m_indptr", "m_indices", "m_data", "out"):
        setattr(a, name, 256)  # the query reads no array
    return a


def _bytes(n, V, grid, precision):
    nbytes = C.c_size_t()
    L.check(L.lib().fm_signal_workspace_size(C.byref(_args(n, V, grid)), PRECISIONS[precision], C.byref(nbytes)))
    return nbytes.value


@pytest.mark.parametrize("precision,real", [("f32", 4), ("f64", 8)])
@pytest.mark.parametrize("V", [1, 8, 32])
@pytest.mark.parametrize("runs", [1, 100, 593, 3000, 6001, 19832])
@pytest.mark.parametrize("slab", [(16, 16), (1, 300), (3, 1)])
def test_partial_sums_of_the_cuda_core_forms(precision, real, V, runs, slab):
    """At most 256 MB more than one node needs, beside the nodes' own arrays (M Mxy
    and the matrix by rows)."""
    n = 200_000
    more = _bytes(n, V, (runs, *slab), precision) - _bytes(1, V, (runs, *slab), precision)
    assert more <= n * (2 * V * real + 16) + 257 * MB


@pytest.mark.parametrize("V", [1, 2, 4])
@pytest.mark.parametrize("grid", [(8, 8, 4), (256, 8, 8), (64, 64, 8)])
@pytest.mark.parametrize("n", [1, 300, 2000])
def test_partial_sums_of_small_tensor_core_problems(n, grid, V):
    """Few nodes: no more than 16 splits' sums, as a served request is counted."""
    S = grid[0] * grid[1] * grid[2]
    assert _bytes(n, V, grid, "bf16x3") <= 16 * S * V * 8 + 64 * S + n * (16 * V + 32) + MB


def test_unfactored_fp64_tiles_are_split_evenly():
    """512 tiles are up to 4 for an SM, or 7 halves: two splits' sums are held."""
    grid, n, V = (16, 8192, 1), 2003, 1
    S = grid[0] * grid[1]
    assert _bytes(n, V, grid, "f64") - _bytes(1, V, grid, "f64") >= 2 * S * V * 16
