"""Rounding errors of the FP32 engines on the grids of up to 64 points, whose x lines (and at 16 and
24 points all lines) run on short plans (Plans in csrc/ns3d_kernels.cuh)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Relative errors of the vorticity of white fields, in units of 1e-7, with one or two long codelets
# per line (16; 12 x 2; 4 x 8; 4 x 12; 8 x 8 points), means of 40 fields: the short plans may not
# round more than those.
LONG_PLANS = {16: 1.066, 24: 1.375, 32: 1.291, 48: 1.529, 64: 1.422}


@pytest.mark.parametrize("N", sorted(LONG_PLANS))
def test_short_plans_round_no_more(ns3d, N):
    k = np.fft.fftfreq(N, 1.0 / N)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + np.arange(N // 2 + 1)[None, None, :] ** 2
    a, b = ns3d.Solver(N), ns3d.Solver(N, precision="fp32")
    errors = []
    for seed in range(16):
        rng = np.random.default_rng(100 * N + seed)
        f = np.fft.rfftn(rng.standard_normal((N, N, N, 3)), axes=(0, 1, 2))
        f[k2 > (N // 3) ** 2] = 0
        f = f.astype(np.complex64).astype(np.complex128)
        a.set_state(f)
        b.set_state(f)
        w, v = a.real_space()[1], b.real_space()[1]
        errors.append(np.linalg.norm((v - w).ravel()) / np.linalg.norm(w.ravel()))
    a.close()
    b.close()
    assert np.mean(errors) < LONG_PLANS[N] * 1e-7
