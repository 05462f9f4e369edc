"""What the integer line transforms of the FP64 engines (csrc/fxfft.cuh, fx_passes.cuh) keep of
double precision: exact zeros, small components beside large ones, the whole range of doubles, and
the rounding errors at every grid size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def wavenumbers(N):
    k = np.array([i if i <= N // 2 else i - N for i in range(N)], dtype=np.float64)
    return k[:, None, None], k[None, :, None], np.arange(N // 2 + 1, dtype=np.float64)[None, None, :]


def white(N, seed=0):
    """Dealiased transform of a white real field [N][N][N/2+1][3]."""
    rng = np.random.default_rng(seed + N)
    f = np.fft.rfftn(rng.standard_normal((N, N, N, 3)), axes=(0, 1, 2))
    kx, ky, kz = wavenumbers(N)
    f[kx * kx + ky * ky + kz * kz > (N // 3) ** 2] = 0
    return f


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("N", [8, 24, 32, 48, 96, 192])
def test_lines_of_zeros(ns3d, N, axis):
    """A flow in a plane stays in it: with no modes along an axis and no velocity in it, the
    term has exact zeros in those modes, as sums of equal numbers have."""
    f = white(N)
    k = wavenumbers(N)[axis]
    f[np.broadcast_to(k != 0, f.shape[:3])] = 0
    f[..., axis] = 0
    s = ns3d.Solver(N, dt=1e-4)
    out = s.NonlinearRHSBatch(f)
    assert np.any(out != 0)
    assert np.all(out[np.broadcast_to(k != 0, f.shape[:3])] == 0)
    s.set_state(f)
    if axis == 2:   # u_z and the vorticity of the plane are lines of their own in every transform
        assert np.all(out[..., 2] == 0)
        u, w = s.real_space()
        assert np.all(u[..., 2] == 0) and np.all(w[..., :2] == 0)
    s.RK4Step(2)
    g = s.get_state()
    assert np.all(g[np.broadcast_to(k != 0, f.shape[:3])] == 0)


# one term of six passes, as in test_fx_fft.py
TOL_RHS = 5e-15
TOL_INV = 2.4e-15


@pytest.mark.parametrize("a", [-500, -480, 480, 495])
@pytest.mark.parametrize("N", [24, 32])
def test_rhs_range(ns3d, N, a):
    """RHS(2^a f) = 2^(2a) RHS(f) as far as the products are normal numbers."""
    f = white(N)
    s = ns3d.Solver(N)
    got = s.NonlinearRHSBatch(f * 2.0 ** a) * 2.0 ** -a
    assert rel(got * 2.0 ** -a, s.NonlinearRHSBatch(f)) < TOL_RHS


@pytest.mark.parametrize("a", [-1000, -955, 905, 1005])
@pytest.mark.parametrize("N", [24, 32])
def test_real_space_range(ns3d, N, a):
    f = white(N)
    s = ns3d.Solver(N)
    s.set_state(f * 2.0 ** a)
    got = s.real_space()
    s.set_state(f)
    for x, y in zip(got, s.real_space()):
        assert rel(x * 2.0 ** (-a // 2) * 2.0 ** (-a - -a // 2), y) < TOL_INV


@pytest.mark.parametrize("a", [-1040, -1060, -1072])
def test_subnormal_fields(ns3d, a):
    """Subnormal modes: the transform keeps their bits and rounds its results once (to within
    one of the spacing, half of it for the double-rounded conversion)."""
    N = 32
    f = white(N) * 2.0 ** a          # cut to multiples of 2^-1074
    s = ns3d.Solver(N)
    s.set_state(f)
    u, _ = s.real_space()
    big = (f * 2.0 ** 600) * 2.0 ** (-a - 600)
    ref = np.fft.irfftn(big, s=(N, N, N), axes=(0, 1, 2)) * 2.0 ** (a + 1074)
    assert np.abs(u[:, :, :N] * 2.0 ** 600 * 2.0 ** 474 - ref).max() <= 1.0
    assert np.any(u != 0) or a < -1065


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("N", [24, 32, 96, 192])
def test_small_component_real_space(ns3d, N, axis):
    """A velocity component far below the others comes back with its own bits."""
    f = white(N)
    f[..., axis] *= 1e-10
    s = ns3d.Solver(N)
    s.set_state(f)
    u, _ = s.real_space()
    ref = np.fft.irfftn(f, s=(N, N, N), axes=(0, 1, 2))
    for c in range(3):
        assert rel(u[:, :, :N, c], ref[..., c]) < TOL_INV, c


@pytest.mark.parametrize("N", [24, 32, 96, 192])
def test_small_component_of_a_plane_flow(ns3d, N):
    """A small velocity across the plane of a two-dimensional flow is advected like a scalar:
    N_z = u_x w_y - u_y w_x is small itself and has its own bits. (The term's sums are products
    of the small field with the large one, so that TOL_RHS holds component by component.)"""
    f = white(N)
    f[:, :, 1:] = 0
    f[..., 2] *= 1e-10
    s = ns3d.Solver(N)
    got = s.NonlinearRHSBatch(f)
    s.set_state(f)
    u, w = s.real_space()
    kx, ky, kz = wavenumbers(N)
    curl = 1j * np.stack([ky * f[..., 2], -kx * f[..., 2], kx * f[..., 1] - ky * f[..., 0]], -1)
    ur = np.fft.ifft2(f[:, :, 0], axes=(0, 1)).real / N
    wr = np.fft.ifft2(curl[:, :, 0], axes=(0, 1)).real / N
    for c in range(3):
        assert rel(u[:, :, 3, c], ur[..., c]) < TOL_INV and rel(w[:, :, 3, c], wr[..., c]) < TOL_INV, c
    nz = np.fft.fft2(ur[..., 0] * wr[..., 1] - ur[..., 1] * wr[..., 0]) * N
    nz[(kx ** 2 + ky ** 2)[..., 0] > (N // 3) ** 2] = 0
    nz[0, 0] = 0
    assert rel(got[:, :, 0, 2], nz) < TOL_RHS
