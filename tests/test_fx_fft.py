"""FP64 engines transform their lines in 64-bit block fixed point (csrc/fxfft.cuh,
fx_passes.cuh): accuracy over the grid sizes' plans, over fields whose lines have
very different ratios of L1 norm to largest value, over the exponent range, and
the lines that hold nothing, too little or a NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# One pass: at most one unit of 2^-61 of a line's L1 norm per input and twiddle product,
# with L1 <= sqrt(2 N) L2, is 2 N 2^-61 (N <= 192: 1.7e-16) of the result's L2 norm for
# the inputs and as much for each of up to three twiddle stages; 1.1e-16 for the rounding
# of its outputs. Three passes stay below 2.4e-15, six (and the product) below 5e-15.
TOL_INV = 2.4e-15
TOL_RHS = 5e-15


def wavenumbers(N):
    k = np.array([i if i <= N // 2 else i - N for i in range(N)], dtype=np.float64)
    return k[:, None, None], k[None, :, None], np.arange(N // 2 + 1, dtype=np.float64)[None, None, :]


def field(N, kind):
    """Dealiased transform of a real field [N][N][N/2+1][3]."""
    rng = np.random.default_rng(N)
    f = np.fft.rfftn(rng.standard_normal((N, N, N, 3)), axes=(0, 1, 2))
    kx, ky, kz = wavenumbers(N)
    k2 = kx * kx + ky * ky + kz * kz
    if kind == "decaying":
        f *= np.exp(-0.5 * np.sqrt(k2))[..., None]
    elif kind == "one mode":
        f *= (k2 == 1)[..., None]
    f[k2 > (N // 3) ** 2] = 0
    return f


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("kind", ["white", "decaying", "one mode"])
@pytest.mark.parametrize("N", [8, 16, 24, 32, 48, 64, 96, 128, 192])
def test_inverse(ns3d, N, kind):
    f = field(N, kind)
    s = ns3d.Solver(N)
    s.set_state(f)
    u, w = s.real_space()
    kx, ky, kz = wavenumbers(N)
    curl = 1j * np.stack([ky * f[..., 2] - kz * f[..., 1], kz * f[..., 0] - kx * f[..., 2],
                          kx * f[..., 1] - ky * f[..., 0]], -1)
    assert rel(u[:, :, :N], np.fft.irfftn(f, s=(N, N, N), axes=(0, 1, 2))) < TOL_INV
    assert rel(w[:, :, :N], np.fft.irfftn(curl, s=(N, N, N), axes=(0, 1, 2))) < TOL_INV


@pytest.mark.parametrize("kind", ["white", "decaying"])
@pytest.mark.parametrize("N", [8, 16, 24, 32, 48, 64])
def test_rhs(ns3d, oracle, N, kind):
    f = field(N, kind)
    assert rel(ns3d.Solver(N).NonlinearRHSBatch(f), oracle.Oracle(N).rhs(f)) < TOL_RHS


@pytest.mark.parametrize("N", [24, 64])
@pytest.mark.parametrize("a", [-400, -130, -60, 0, 60, 130, 400])
def test_rhs_over_the_exponent_range(ns3d, N, a):
    """RHS(2^a f) = 2^(2a) RHS(f), also where a line's bound leaves FP32's range."""
    f = field(N, "decaying")
    s = ns3d.Solver(N)
    base = s.NonlinearRHSBatch(f)
    assert rel(s.NonlinearRHSBatch(f * 2.0 ** a) * 2.0 ** (-2 * a), base) < TOL_RHS


def test_lines_out_of_the_exponent_range(ns3d):
    f = field(32, "white")
    s = ns3d.Solver(32)
    assert np.all(s.NonlinearRHSBatch(np.zeros_like(f)) == 0)
    assert np.all(s.NonlinearRHSBatch(f * 2.0 ** -980) == 0)       # taken as zero
    assert np.all(s.NonlinearRHSBatch(f * 2.0 ** -560) == 0)       # the products are
    assert not np.any(np.isfinite(s.NonlinearRHSBatch(f * 2.0 ** 600)[1, 1, 1]))   # the products overflow
    ok = s.NonlinearRHSBatch(f)
    assert np.all(np.isfinite(ok)) and np.any(ok != 0)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_nan_and_inf(ns3d, bad):
    f = field(32, "white")
    f[2, 3, 4, 1] = bad
    s = ns3d.Solver(32, dt=1e-3)
    assert np.any(np.isnan(s.NonlinearRHSBatch(f)))
    s.set_state(f)
    with pytest.raises(ns3d.NS3DError) as e:
        s.RK4Step(2)
    assert e.value.status == ns3d.ERR_NUMERIC
