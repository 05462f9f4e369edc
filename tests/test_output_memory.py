"""What the real-space output leaves allocated: the staging buffer of a large grid is given back."""
import pytest

pytestmark = pytest.mark.gpu


def test_real_space_gives_its_staging_back(ns3d):
    import torch
    N = 256
    with ns3d.Solver(N, precision="fp32") as s:
        # the initial condition allocates the context's real fields; no state crosses the link, so
        # nothing is staged yet
        s.InitialConditions("TAYLOR_GREEN")
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s.real_space()
        after = torch.cuda.mem_get_info()[0]
        assert before - after < 64 << 20
        s.real_space()
        assert torch.cuda.mem_get_info()[0] >= after - (4 << 20)
