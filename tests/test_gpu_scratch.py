"""Scratch of the reductions grows with a lane's largest basis, not with the largest there is."""
import pytest

import molds_gb300 as M

pytestmark = pytest.mark.gpu


def test_small_lane_scratch():
    """4096 slots of up to 64 basis functions: 0.2 KB of DIIS sums, 2.1 KB of energy and
    dipole sums, 0.5 KB of purification state and under 3 KB of lists and records each."""
    ctx = M.Context(0)
    srv = M.Server(M.SCFParams(), context=ctx, hbm_budget_bytes=64 << 20, max_basis=64)
    used = srv.device_bytes()
    srv.close()
    ctx.close()
    assert used <= (64 << 20) + 4096 * 6144
