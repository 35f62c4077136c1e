"""Lone atoms: no gap in any iteration, so every density is the eigensolver's and
none of their iterations waits for it."""
import numpy as np
import pytest

import molds_gb300 as M
from molds_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = M.Context(0)
    yield c
    c.close()


def _atom(z):
    return M.Molecule(np.array([z], dtype=np.int32), np.zeros((1, 3)))


@pytest.mark.parametrize("z", [6, 8, 16])
def test_atom_needs_no_more_iterations_than_with_the_eigensolver(ctx, z):
    out = []
    for solver in ("auto", "householder"):
        b = M.ResidentBatch("pm3", [_atom(z)], context=ctx)
        b.run(M.SCFParams(eigensolver=solver))
        res, q = b.results()
        out.append((res[0]["status"], res[0]["iterations"], res[0]["energy"], b.graph_launch_count()))
        b.close()
    assert out[0] == out[1]
    assert out[0][0] == M.STATUS_CONVERGED


def test_repeated_runs_replay_one_graph_per_iteration(ctx):
    """A second run with the same settings replays as many iterations as the first, for either solver."""
    for solver in ("auto", "householder"):
        b = M.ResidentBatch("pm3", [_atom(8), _atom(16)], context=ctx)
        counts = []
        for _ in range(2):
            before = b.graph_launch_count()
            b.run(M.SCFParams(eigensolver=solver))
            counts.append(b.graph_launch_count() - before)
        b.close()
        assert counts[0] == counts[1]


def test_atom_beside_molecules(ctx):
    """The same bits as alone, for the atom and for its neighbours of either kernel."""
    prm = M.SCFParams(damping_weight=0.0, diis_start_error=0.1, diis_end_error=0.0)
    mols = [W.water_cluster_k(4, 3), _atom(8), W.water_cluster_k(25, 3)]
    both, q = M.batch_scf("am1", mols, prm, context=ctx)
    for i, m in enumerate(mols):
        alone, qa = M.batch_scf("am1", [m], prm, context=ctx)
        assert both[i]["status"] == alone[0]["status"] == M.STATUS_CONVERGED
        assert both[i]["energy"] == alone[0]["energy"] and both[i]["iterations"] == alone[0]["iterations"]
        assert np.array_equal(q[i], qa[0])


def test_served_atom(ctx):
    prm = M.SCFParams()
    alone, _ = M.batch_scf("pm3", [_atom(8)], prm, context=ctx)
    srv = M.Server(prm, context=ctx, hbm_budget_bytes=1 << 30, max_basis=64)
    try:
        srv.submit("pm3", _atom(8))
        r = []
        for _ in range(1000):
            r += srv.poll(max_wait_us=10000)
            if r:
                break
    finally:
        srv.close()
    assert len(r) == 1 and r[0]["status"] == M.STATUS_CONVERGED
    assert r[0]["energy"] == alone[0]["energy"] and r[0]["iterations"] == alone[0]["iterations"]
