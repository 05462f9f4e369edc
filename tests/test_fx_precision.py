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


def plane_flow(N):
    """White flow in the x-z plane: transforms [N][N/2+1] of u_x and u_z (u_y = 0, no y dependence)."""
    rng = np.random.default_rng(N)
    k = np.fft.fftfreq(N, 1.0 / N)[:, None]
    kz = np.arange(N // 2 + 1, dtype=np.float64)[None, :]
    keep = k * k + kz * kz <= (N // 3) ** 2
    return [np.fft.rfft2(rng.standard_normal((N, N))) * keep for _ in range(2)], k, kz, keep


def check_plane_flow(ns3d, N):
    """Real space and the right-hand side against transforms in extended precision. Tolerance: one
    unit of 2^-53 per radix-2 level, the levels' errors independent: two inverse transforms for a
    field, and those of both factors and two forward ones for the term."""
    sfft = pytest.importorskip("scipy.fft")
    unit = 2.0 ** -53 * np.sqrt(np.log2(N))
    (fx, fz), k, kz, keep = plane_flow(N)
    f = np.zeros((N, N, N // 2 + 1, 3), np.complex128)
    f[:, 0, :, 0], f[:, 0, :, 2] = fx * N, fz * N
    s = ns3d.Solver(N)
    got = s.NonlinearRHSBatch(f)[:, 0].copy()
    s.set_state(f)
    del f
    u, w = (a[:, 5, :N].copy() for a in s.real_space())
    s.close()
    fx, fz = fx.astype(np.clongdouble), fz.astype(np.clongdouble)
    ux, uz, wy = (sfft.irfft2(a, s=(N, N)) for a in (fx, fz, 1j * (kz * fx - k * fz)))
    for a, b in ((u[..., 0], ux), (u[..., 2], uz), (w[..., 1], wy)):
        assert rel(a, b) < unit * np.sqrt(2)
    nx, nz = sfft.rfft2(-uz * wy), sfft.rfft2(ux * wy)
    k2 = np.where(keep & (k * k + kz * kz > 0), k * k + kz * kz, np.inf)
    d = (k * nx + kz * nz) / k2
    ref = np.stack([(n - q * d) * np.isfinite(k2) * N for n, q in ((nx, k), (nz, kz))], -1)
    assert np.all(got[..., 1] == 0)
    assert rel(got[..., ::2], ref) < unit * np.sqrt(6)


@pytest.mark.parametrize("N", [24, 64, 128, 192, 256, 384, 512, 768])
def test_plane_flow(ns3d, N):
    check_plane_flow(ns3d, N)


@pytest.mark.parametrize("N", [128, 192, 256, 384, 512, 768])
def test_against_device_transforms(ns3d, N):
    """White fields through every pass (real space, the right-hand side, real space back to modes),
    component by component, against FP64 transforms of the device library. Tolerance as in
    test_plane_flow, three transforms per field and nine for the term, of both sides."""
    import torch
    unit = 2 * 2.0 ** -53 * np.sqrt(np.log2(N))
    gen = torch.Generator(device="cuda").manual_seed(N)
    k = torch.fft.fftfreq(N, 1.0 / N, dtype=torch.float64, device="cuda")
    ks = (k[:, None, None], k[None, :, None], torch.arange(N // 2 + 1, dtype=torch.float64, device="cuda"))
    keep = ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2 <= (N // 3) ** 2
    f = [torch.fft.rfftn(torch.randn(N, N, N, dtype=torch.float64, device="cuda", generator=gen)) * keep for _ in range(3)]
    host = torch.stack(f, -1).cpu().numpy()
    s = ns3d.Solver(N)
    got = s.NonlinearRHSBatch(host)
    s.set_state(host)
    del host
    u, w = s.real_space()
    s.set_state_real(u)
    back = s.get_state()
    s.close()

    def err(a, b):
        return float((torch.from_numpy(np.ascontiguousarray(a)).cuda() - b).norm() / b.norm())

    ur = [torch.fft.irfftn(a, s=(N, N, N)) for a in f]
    wr = []
    for c in range(3):
        a, b = (c + 1) % 3, (c + 2) % 3
        wr.append(torch.fft.irfftn(1j * (ks[a] * f[b] - ks[b] * f[a]), s=(N, N, N)))
    for c in range(3):
        assert err(u[:, :, :N, c], ur[c]) < unit * np.sqrt(3), c
        assert err(w[:, :, :N, c], wr[c]) < unit * np.sqrt(3), c
        assert err(back[..., c], f[c]) < unit * np.sqrt(6), c
    del u, w, back
    n = [torch.fft.rfftn(ur[(c + 1) % 3] * wr[(c + 2) % 3] - ur[(c + 2) % 3] * wr[(c + 1) % 3]) for c in range(3)]
    del ur, wr
    k2 = (ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2)
    d = sum(ks[c] * n[c] for c in range(3)) / k2.clamp(min=1)
    for c in range(3):
        assert err(got[..., c], (n[c] - ks[c] * d) * keep * (k2 > 0)) < unit * 3, c


def test_stage_weights_are_rounded_once(ns3d):
    """The IF-RK4 weights h / 6 and h / 3 are the nearest doubles. With a step h whose sixth rounds to
    2e-17, while the product h (1 / 6) is off by 9e-17, the error of one step's increment along
    itself tells the two apart: the other errors are random over the modes."""
    sfft = pytest.importorskip("scipy.fft")
    from fractions import Fraction as F
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision")
    N = 48
    (fx, fz), k, kz, keep = plane_flow(N)
    k2 = np.where(keep & (k * k + kz * kz > 0), k * k + kz * kz, np.inf)
    d = (k * fx + kz * fz) / k2
    fx, fz = (fx - k * d) * np.isfinite(k2), (fz - kz * d) * np.isfinite(k2)

    def rhs(a):
        ux, uz, wy = (sfft.irfft2(q, s=(N, N)) for q in (a[0], a[1], 1j * (kz * a[0] - k * a[1])))
        n = [sfft.rfft2(-uz * wy), sfft.rfft2(ux * wy)]
        e = (k * n[0] + kz * n[1]) / k2
        return np.stack([(n[0] - k * e) * np.isfinite(k2), (n[1] - kz * e) * np.isfinite(k2)])

    u = np.stack([fx, fz])
    scale = np.linalg.norm(u.ravel()) / np.linalg.norm(rhs(u).ravel())
    rng = np.random.default_rng(0)
    best, h = 0, None
    for c in scale * rng.uniform(0.7, 1.0, 20000):
        six = F(float(c)) / 6
        off = [abs(float((F(q) - six) / six)) for q in (float(c) * (1.0 / 6.0), float(c) / 6.0)]
        if off[0] - off[1] > best:
            best, h = off[0] - off[1], float(c)
    assert best > 7e-17
    f = np.zeros((N, N, N // 2 + 1, 3), np.complex128)
    f[:, 0, :, 0], f[:, 0, :, 2] = fx * N, fz * N
    s = ns3d.Solver(N, nu=1e-30, dt=h, integrator="ifrk4")
    s.set_state(f)
    s.RK4Step(1)
    g = s.get_state()[:, 0]
    s.close()
    u, h = u.astype(np.clongdouble), np.longdouble(h)
    k1 = rhs(u)
    k2_ = rhs(u + h / 2 * k1)
    k3 = rhs(u + h / 2 * k2_)
    step = h / 6 * (k1 + 2 * k2_ + 2 * k3 + rhs(u + h * k3))
    err = np.stack([g[..., 0], g[..., 2]]) / N - (u + step)
    slope = float(np.sum((err * np.conj(step)).real) / np.sum(np.abs(step) ** 2))
    assert abs(slope) < 5e-17
