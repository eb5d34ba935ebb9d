"""Steps whose field does not change: segments of every length without RF, with
one gradient or none, against the same steps one solve at a time, whose single
steps have no such segment.  Bit for bit; and nodes or motion at no finite place
stay not a number."""
import numpy as np
import pytest

from feelmri_b200 import workloads as W
from feelmri_b200.BlochSimulator import solve_mri

pytestmark = pytest.mark.gpu


def _steps(seed):
    """Runs of 1 .. 9 steps: RF on or off, gradients held, zero or changing."""
    rng = np.random.default_rng(seed)
    rf, G, dt = [0j], [(0, 0, 0)], [0.0]
    for _ in range(40):
        n, on, kind, d = rng.integers(1, 10), rng.random() < 0.2, rng.integers(0, 3), rng.choice([0.01, 0.5])
        g = rng.normal(0, 5.0, 3) * (kind > 0)
        for _ in range(n):
            rf.append(complex(*rng.normal(0, 1e-3, 2)) if on else 0j)
            G.append(rng.normal(0, 5.0, 3) if kind == 2 else g)
            dt.append(d)
    c = lambda a, t: np.asarray(a, t)
    return c(rf, np.complex64), c(G, np.float32), c(dt, np.float32)


def _solve(rf, G, dt, r0, Mxy, Mz, dB, T1, T2, pod):
    return solve_mri(r0, T1, T2, dB, 1.0, float(np.float32(W.GAMMA)), rf, G, dt, np.abs(rf) != 0, Mxy, Mz, pod)


@pytest.mark.parametrize("seed", range(3))
def test_static_steps_equal_single_steps(cuda, seed):
    rng = np.random.default_rng(100 + seed)
    n = 130
    rf, G, dt = _steps(seed)
    r0 = rng.uniform(-0.05, 0.05, (n, 3)).astype(np.float32)
    T1 = rng.uniform(800, 1200, n).astype(np.float32)
    T2 = rng.uniform(50, 100, n).astype(np.float32)
    dB = rng.normal(0, 1e-4, n).astype(np.float32)
    dB[:3] = 0.0
    r0[5] = np.nan
    r0[6, 1] = np.inf
    Mxy = (rng.normal(size=n) + 1j * rng.normal(size=n)).astype(np.complex64)
    Mz = rng.uniform(0.2, 1.0, n).astype(np.float32)
    m, z = _solve(rf, G, dt, r0, Mxy, Mz, dB, T1, T2, None)
    for i in range(1, rf.size):
        pick = [0, i]
        a, b = _solve(rf[pick], G[pick], dt[pick], r0, m[:, i - 1].copy(), z[:, i - 1].copy(), dB, T1, T2, None)
        np.testing.assert_array_equal(a[:, 1], m[:, i])
        np.testing.assert_array_equal(b[:, 1], z[:, i])
    assert np.isnan(m[5:7, 1:]).all() and np.isfinite(np.delete(m, [5, 6], 0)).all()


@pytest.mark.parametrize("modes", [1, 4, 7])
def test_moving_steps(cuda, modes):
    """The motion as a lowered term, and sampled as a callable (no segment there).
    Its displacements differ by FP32 rounding between the two, as does the field
    on steps with a gradient."""
    rng = np.random.default_rng(7)
    n = 130
    rf, G, dt = _steps(5)
    pod = W.sinusoidal_pod(n, n_modes=modes, amp=1e-3, period=20.0, n_frames=9)
    r0 = rng.uniform(-0.05, 0.05, (n, 3)).astype(np.float32)
    r0[9] = np.nan
    r0[10, 2] = np.inf
    T1, T2 = np.full(n, 1000, np.float32), np.full(n, 80, np.float32)
    dB = rng.normal(0, 1e-4, n).astype(np.float32)
    Mxy, Mz = np.full(n, 0.3 - 0.2j, np.complex64), np.full(n, 0.7, np.float32)
    m, z = _solve(rf, G, dt, r0, Mxy, Mz, dB, T1, T2, pod)
    mt, zt = _solve(rf, G, dt, r0, Mxy, Mz, dB, T1, T2, lambda t: pod(t))
    bad = np.isin(np.arange(n), [9, 10])
    assert np.isnan(m[bad, 1:]).all() and np.isnan(mt[bad, 1:]).all()
    scale = np.abs(mt[~bad]).max()
    assert np.abs(m[~bad] - mt[~bad]).max() < 1e-4 * scale and np.abs(z[~bad] - zt[~bad]).max() < 1e-4
    # a motion that is not a number leaves nothing a number, gradient or not
    pod.update_timeshift(np.float32(np.nan))
    m, z = _solve(rf, 0 * G, dt, r0, Mxy, Mz, dB, T1, T2, pod)
    assert np.isnan(m[:, 1:]).all()


@pytest.mark.parametrize("n", [1, 129, 148 * 128, 148 * 128 + 1])
def test_one_launch_and_two(cuda, n):
    """257 steps are prepared by their own launch, the first 256 of them (up to
    148 blocks of nodes) within the sweep: the same bits."""
    rng = np.random.default_rng(11)
    rf, G, dt = (np.concatenate([a, a[1:], a[1:]]) for a in _steps(4))
    rf, G, dt = rf[:258], G[:258], dt[:258]
    assert rf.size == 258
    r0 = rng.uniform(-0.05, 0.05, (n, 3)).astype(np.float32)
    T1, T2 = np.full(n, 1000, np.float32), np.full(n, 80, np.float32)
    dB = rng.normal(0, 1e-4, n).astype(np.float32)
    Mxy, Mz = np.full(n, 0.3 - 0.2j, np.complex64), np.full(n, 0.7, np.float32)
    m, z = _solve(rf, G, dt, r0, Mxy, Mz, dB, T1, T2, None)
    a, b = _solve(rf[:257], G[:257], dt[:257], r0, Mxy, Mz, dB, T1, T2, None)
    np.testing.assert_array_equal(a, m[:, :257])
    np.testing.assert_array_equal(b, z[:, :257])
