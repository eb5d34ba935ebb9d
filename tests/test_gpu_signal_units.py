"""Signal work units at the sizes where they can go wrong, against the FP64
oracle: partial row and column tiles of every unit kind, few rows, node ranges
that end inside a stage or block, the run and sparse-matrix preparation.

Tolerances: the split-BF16 form keeps hi hi + hi lo + lo hi, so a product is
off by at most about 3 x 2^-17 of its size; over incoherent sums that is below
the form's bar of 1e-4 relative L2."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import fp64
from feelmri_b200 import workloads as W
from feelmri_b200.MRI import Signal, signal_call_times

pytestmark = pytest.mark.gpu

TC_TOL = 1e-4


def _case(n, V, seed=0):
    rng = np.random.default_rng(seed)
    r0 = rng.uniform(-0.04, 0.04, (n, 3)).astype(np.float32)
    Mxy = ((rng.normal(size=(n, V)) + 1j * rng.normal(size=(n, V))) * 0.1).astype(np.complex64)
    phi = W.off_resonance(n)
    T2 = rng.uniform(50.0, 100.0, n).astype(np.float32)
    M = sp.diags(rng.uniform(1e-7, 3e-7, n)).tocsc()
    return r0, M, Mxy, phi, T2


def _ref(M, traj, t, r0, phi, T2, Mxy, pod=None):
    disp = None if pod is None else np.stack([pod(x) for x in signal_call_times(t)[1:]])
    return fp64.signal(sp.csc_matrix(M), *traj.points, t, r0, phi, T2, Mxy, disp=disp, pi_mode="float")


def _traj(kind, res):
    if kind == "cartesian":
        return W.cartesian(res=res)
    if kind == "spiral":
        return W.spiral_stack(n_ro=res[0], n_interleaves=res[1], n_kz=res[2])
    return W.radial3d(n_ro=res[0], n_spokes=res[1], kmax=300.0)


@pytest.mark.parametrize("kind,res,V,n,motion", [
    ("cartesian", (5, 16, 8), 1, 700, False),     # runs as columns: 5 runs, one row tile
    ("cartesian", (17, 11, 3), 1, 129, False),    # 17 columns: both node halves apart
    ("cartesian", (33, 7, 5), 2, 513, False),     # 35 rows, 33 runs of 2 columns
    ("cartesian", (70, 13, 4), 1, 300, False),    # 70 runs in one tile, 52 rows
    ("cartesian", (150, 9, 1), 1, 257, False),    # two column tiles, kz = 1
    ("cartesian", (20, 40, 9), 8, 400, False),    # 20 runs of 8 columns: two column tiles
    ("cartesian", (3, 96, 32), 4, 1111, True),    # wide slab, three row groups
    ("cartesian", (3, 33, 40), 3, 600, True),     # 33 rows, 40 kz values
    ("cartesian", (2, 130, 70), 1, 200, True),    # a second row tile of two rows
    ("spiral", (40, 3, 16), 2, 515, False),       # stacked runs
    ("spiral", (9, 20, 17), 1, 100, False),       # stacked, more than 16 kz values
    ("radial", (6, 31, 1), 8, 1030, True),        # generic, one row group
    ("radial", (4, 64, 1), 3, 2050, False),       # generic, two row groups
    ("radial", (3, 300, 1), 9, 130, True),        # generic, two column groups, partial row tile
])
def test_tensor_core_units(cuda, kind, res, V, n, motion):
    r0, M, Mxy, phi, T2 = _case(n, V)
    traj = _traj(kind, res)
    pod = W.sinusoidal_pod(n, n_modes=3, amp=1e-3, period=50.0, n_frames=8) if motion else None
    K = Signal(0, M, traj.points, traj.t, r0, phi, T2, Mxy, pod, precision="bf16x3")
    assert fp64.rel_l2(K, _ref(M, traj, traj.t, r0, phi, T2, Mxy, pod)) < TC_TOL


@pytest.mark.parametrize("precision,tol", [("bf16x3", TC_TOL), (None, 1e-5)])
@pytest.mark.parametrize("what", ["line_times", "sample_times", "merged_runs", "permutation", "shared_rows"])
def test_runs_and_sparse_products(cuda, what, precision, tol):
    """Sample times that do not follow the slabs, and mass matrices of as many
    entries as rows that are not diagonal."""
    n, V = 900, 2
    r0, M, Mxy, phi, T2 = _case(n, V, seed=3)
    traj = W.cartesian(res=(6, 10, 4))
    t = traj.t.copy()
    rng = np.random.default_rng(5)
    if what == "line_times":
        t += (np.arange(10, dtype=np.float32) * 0.001)[None, :, None]
    elif what == "sample_times":
        t = (2.0 + 0.001 * np.arange(t.size, dtype=np.float32)).reshape(t.shape)
    elif what == "merged_runs":
        t[2] = t[1]  # two slabs are one run
        t[4, 5:] += np.float32(0.01)  # one slab is two
    elif what == "permutation":
        M = sp.csc_matrix((M.diagonal(), (rng.permutation(n), np.arange(n))), shape=(n, n))
    else:  # n entries, several in one row, some columns empty
        M = sp.csc_matrix((M.diagonal(), (rng.integers(0, n, n), np.sort(rng.integers(0, n, n)))), shape=(n, n))
    K = Signal(0, M, traj.points, t, r0, phi, T2, Mxy, None, precision=precision)
    assert fp64.rel_l2(K, _ref(M, traj, t, r0, phi, T2, Mxy)) < tol


# CUDA-core forms whose samples factor: rounding of the FP64 form is some 1e-15 a
# term and does not add up coherently over these few nodes; FP32 has the bar of
# its drop-in form.
@pytest.mark.parametrize("precision,tol", [("f64", 1e-13), (None, 1e-5)])
@pytest.mark.parametrize("res,V,n,motion", [
    ((2, 3, 1), 1, 17, False),      # one thread's rows and columns
    ((64, 64, 1), 1, 700, False),   # one full tile (FP64)
    ((65, 9, 1), 1, 129, False),    # a second column tile of one column
    ((7, 43, 3), 3, 515, False),    # 129 rows: a second row tile of one
    ((5, 11, 2), 70, 65, False),    # more columns per run than a tile holds
    ((4, 6, 5), 13, 33, True),      # 65 columns of 13 weights
    ((3, 131, 2), 2, 301, True),    # three row tiles
    ((2, 2, 80), 1, 1, True),       # one node
    ((3, 5, 16), 4, 2049, True),    # stage ends
    ((1, 40, 6), 2, 500, False),    # one run: slabs
])
def test_factored_forms(cuda, res, V, n, motion, precision, tol):
    r0, M, Mxy, phi, T2 = _case(n, V)
    traj = _traj("cartesian", res)
    pod = W.sinusoidal_pod(n, n_modes=3, amp=1e-3, period=50.0, n_frames=8) if motion else None
    pts, t = traj.points, traj.t
    if precision == "f64":
        r0, phi, T2, t = (a.astype(np.float64) for a in (r0, phi, T2, t))
        pts = tuple(np.asarray(p, np.float64) for p in pts)
        Mxy = Mxy.astype(np.complex128)
    K = Signal(0, M, pts, t, r0, phi, T2, Mxy, pod)
    assert K.dtype == Mxy.dtype
    ref = fp64.signal(sp.csc_matrix(M), *pts, t, r0, phi, T2, Mxy, pi_mode="float",
                      disp=None if pod is None else np.stack([pod(x) for x in signal_call_times(t)[1:]]))
    # displacements are FP32 numbers in both
    assert fp64.rel_l2(K, ref) < (tol if pod is None or precision is None else 1e-6)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_factored_forms_far_and_not_finite(cuda, dtype):
    """Phases of millions of cycles, and nodes at no finite place."""
    n = 80
    r0, M, Mxy, phi, T2 = _case(n, 1)
    traj = W.cartesian(res=(4, 6, 3))
    c = lambda a: np.asarray(a, dtype)
    pts = [c(p) for p in traj.points]
    pts[1] = c(np.float32(pts[1] * 1e6))
    args = (c(traj.t), c(r0), c(phi), c(T2), Mxy.astype(np.complex64 if dtype == np.float32 else np.complex128))
    K = Signal(0, M, tuple(pts), *args, None)
    ref = fp64.signal(sp.csc_matrix(M), *pts, *args, disp=None, pi_mode="float")
    assert fp64.rel_l2(K, ref) < 1e-5
    for bad in (np.nan, np.inf):
        r1 = args[1].copy()
        r1[3, 2] = bad
        assert np.isnan(Signal(0, M, tuple(pts), args[0], r1, *args[2:], None)).all()


# The unfactored FP32 form at the edges of its tiles of 256 samples, node stages
# of 128 and column groups of 8; phases of millions of cycles; nodes at no finite
# place.  Its drop-in form's bar.
@pytest.mark.parametrize("res,V,n,motion", [
    ((1, 1, 1), 1, 1, False),
    ((3, 128, 1), 2, 127, False),
    ((3, 129, 1), 3, 129, True),
    ((2, 256, 1), 8, 256, False),
    ((2, 257, 1), 9, 2049, True),
    ((1, 700, 1), 5, 1500, False),
])
def test_unfactored_form(cuda, res, V, n, motion):
    r0, M, Mxy, phi, T2 = _case(n, V)
    traj = _traj("radial", res)
    pod = W.sinusoidal_pod(n, n_modes=3, amp=1e-3, period=50.0, n_frames=8) if motion else None
    pts = [np.asarray(p, np.float32) for p in traj.points]
    for scale in (1.0, 1e6):
        k = (pts[0], np.float32(pts[1] * scale), pts[2])
        K = Signal(0, M, k, traj.t, r0, phi, T2, Mxy, pod)
        ref = fp64.signal(sp.csc_matrix(M), *k, traj.t, r0, phi, T2, Mxy, pi_mode="float",
                          disp=None if pod is None else np.stack([pod(x) for x in signal_call_times(traj.t)[1:]]))
        if scale == 1.0 or pod is None:  # the displaced place is rounded to FP32
            assert fp64.rel_l2(K, ref) < 1e-5
    for bad in (np.nan, np.inf):
        r1 = r0.copy()
        r1[0, 1] = bad
        assert np.isnan(Signal(0, M, traj.points, traj.t, r1, phi, T2, Mxy, pod)).all()


@pytest.mark.parametrize("kind,res,dtype,tol", [
    ("cartesian", (600, 8, 2), np.float32, 1e-5),  # factored
    ("cartesian", (600, 8, 2), np.float64, 1e-6),  # displacements are FP32 numbers
    ("radial", (600, 40, 1), np.float32, 1e-5),    # unfactored
])
def test_sums_cut_within_a_node_range(cuda, kind, res, dtype, tol):
    """So many runs that a node range is longer than one sum in registers."""
    n, V = 12000, 2
    r0, M, Mxy, phi, T2 = _case(n, V)
    traj = _traj(kind, res)
    pod = W.sinusoidal_pod(n, n_modes=2, amp=1e-3, period=50.0, n_frames=8)
    c = lambda a: np.asarray(a, dtype)
    pts, args = tuple(c(p) for p in traj.points), (c(traj.t), c(r0), c(phi), c(T2))
    K = Signal(0, M, pts, *args, Mxy.astype(np.complex64 if dtype == np.float32 else np.complex128), pod)
    pick = np.random.default_rng(2).permutation(traj.t.size)[:300]
    disp = np.stack([pod(x) for x in signal_call_times(args[0])[1:]])
    ref = fp64.signal(sp.csc_matrix(M), *pts, *args, Mxy, pi_mode="float", disp=disp, sample_idx=pick)
    assert fp64.rel_l2(K.reshape(-1, V)[pick], ref) < tol
