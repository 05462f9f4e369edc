"""Transform plans and x tiles of small grids: the FP32 right-hand side over the sizes with
short plans, and members of groups on both sides of the tile rule (x_small in
csrc/ns3d_kernels.cuh), whose transforms are the same as a single run's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 24, 48])
def test_rhs_fp32_small(ns3d, oracle, N):
    # each of the six passes loses at most 6 units of 2^-24 per radix-2 level in the L2 norm;
    # the projection of u x w may cancel up to a factor of 4 of its norm on these fields
    tol = 4 * 6 * 6 * np.log2(N) * 2.0 ** -24
    rng = np.random.default_rng(N)
    f = np.fft.rfftn(rng.standard_normal((N, N, N, 3)), axes=(0, 1, 2))
    k = np.fft.fftfreq(N, 1.0 / N)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + np.arange(N // 2 + 1)[None, None, :] ** 2
    f[k2 > (N // 3) ** 2] = 0
    f = f.astype(np.complex64).astype(np.complex128)
    r = oracle.Oracle(N).rhs(f)
    g = ns3d.Solver(N, precision="fp32").NonlinearRHSBatch(f)
    assert np.linalg.norm((g - r).ravel()) < tol * np.linalg.norm(r.ravel())


@pytest.mark.parametrize("N,members,prec", [(32, 5, "fp32"), (48, 8, "fp32"), (48, 9, "fp32"), (64, 9, "fp32"),
                                            (96, 3, "fp32"), (96, 5, "fp32"), (128, 2, "fp32"),
                                            (24, 9, "fp64"), (32, 9, "fp64"), (48, 3, "fp64")])
def test_group_members_equal_single_runs(ns3d, N, members, prec):
    par = [dict(N=N, nu=0.01 / (1 + i), dt=1e-3, precision=prec) for i in range(members)]
    ens = ns3d.Ensemble(par)
    for i in range(members):
        ens.InitialConditions(i, "SPECTRUM", seed=5 + i, k0=3.0)
    ens.step(2)
    for i in (0, members - 1):
        s = ns3d.Solver(**par[i])
        s.InitialConditions("SPECTRUM", seed=5 + i, k0=3.0)
        s.RK4Step(2)
        assert np.array_equal(ens.get_state(i), s.get_state()), i
        s.close()
    ens.close()
