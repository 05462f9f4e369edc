"""The per-kernel profile names the kernels that run and counts their bytes in both precisions."""
import pytest

pytestmark = pytest.mark.gpu


def test_profile_names_and_bytes(ns3d):
    N, rows = 32, {}
    for prec in ("fp32", "fp64"):
        with ns3d.Solver(N, precision=prec) as s:
            s.InitialConditions("TAYLOR_GREEN")
            rows[prec] = s.profile_step(1)
    assert [r[0] for r in rows["fp64"]] == ["k_xinv_fx", "k_ypass_fx_inv", "k_zfx", "k_ypass_fx_fwd", "k_xfwd_fx", "k_misc"]
    # twice the FP32 bytes, and four bytes per line for its scale: three z lines per (x, y), six
    # lines read per (x, kz)
    extra = [b64 - 2 * b32 for (_, _, b32), (_, _, b64) in zip(rows["fp32"], rows["fp64"])]
    assert extra[2] == 4 * (3 * N * N + 6 * N * (N // 3 + 1))
    assert all(e > 0 for e in extra[:5]) and extra[5] == 0
