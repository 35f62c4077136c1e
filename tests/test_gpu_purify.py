"""Density by purification (csrc/purify.cu) against numpy's eigenvectors of the
oracle's guess Fock matrix, at the edges of its kernels: the one-CTA kernel's
column halves (64) and padding (16), its limit (128), the tile kernel's row and
column tiles (128, 64), its padding (32) and its K segments (1024).  And the
molecules it hands to the eigensolver."""
import numpy as np
import pytest

import molds_gb300 as M
from molds_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ANG = M.ANG2AU


@pytest.fixture(scope="module")
def ctx():
    c = M.Context(0)
    yield c
    c.close()


def _molecule(n, seed):
    """Waters (6 basis functions) and H2 (2) on a jittered lattice: n basis functions, n even."""
    h2 = (n % 6) // 2 if n >= 6 else n // 2
    k = (n - 2 * h2) // 6
    side = int(np.ceil((k + h2) ** (1.0 / 3.0)))
    rng = np.random.default_rng(seed)
    Z, xyz = [], []
    sites = [(i, j, l) for i in range(side) for j in range(side) for l in range(side)][:k + h2]
    for m, s in enumerate(sites):
        c = np.array(s) * 2.9 + rng.uniform(-0.2, 0.2, 3)
        u = rng.normal(size=(2, 3))
        u /= np.linalg.norm(u, axis=1)[:, None]
        if m < k:
            Z += [8, 1, 1]
            xyz += [c, c + 0.96 * u[0], c + 0.96 * np.cross(u[0], u[1]) / np.linalg.norm(np.cross(u[0], u[1]))]
        else:
            Z += [1, 1]
            xyz += [c, c + 0.74 * u[0]]
    return M.Molecule(np.array(Z, dtype=np.int32), np.array(xyz) * ANG)


@pytest.mark.parametrize("n", [2, 16, 18, 62, 64, 66, 112, 128, 130, 160, 162, 192, 194, 256, 258, 384, 1024, 1030])
def test_guess_density(ctx, n):
    mol = _molecule(n, n)
    es = M.ElectronicStructure("am1", M.SCFParams(max_iter=1), context=ctx)
    es.SetMolecule(mol)
    with pytest.raises(M.SCFNotConverged):
        es.DoSCF(True)
    P = es.GetOrbitalElectronPopulation()
    m = O.make_molecule("am1", mol.Z, mol.xyz)
    S, eri, _ = O.integrals(m)
    F = O.fock(m, S, eri, np.zeros((n, n)), guess=True)
    w, v = np.linalg.eigh(F)
    nocc = int(round(O.atom_info(m)[:, 0].sum())) // 2
    ref = 2.0 * v[:, :nocc] @ v[:, :nocc].T
    # numpy's projector is off by about n eps ||F|| / gap; five times that
    tol = max(1e-14, 5 * n * 2.2e-16 * np.abs(w).max() / (w[nocc] - w[nocc - 1]))
    assert P.shape == (n, n) and np.abs(P - ref).max() <= tol
    assert np.array_equal(P, P.T)
    # idempotent to the rounding of the product that checks it
    assert np.abs(0.5 * P @ P - P).max() <= 4 * n * 2.2e-16 + 2e-15


def _degenerate(waters):
    """A water cluster and a lone oxygen atom far away: three degenerate p orbitals, two of them occupied."""
    mol = W.water_cluster_k(waters, 5) if waters else M.Molecule(np.zeros(0, dtype=np.int32), np.zeros((0, 3)))
    xyz = np.concatenate([mol.xyz.reshape(-1, 3), [[400.0, 410.0, 420.0]]])
    return M.Molecule(np.concatenate([mol.Z, [8]]).astype(np.int32), xyz)


@pytest.mark.parametrize("waters", [0, 3, 15, 25])
def test_degenerate_frontier_takes_the_eigensolver(ctx, waters):
    """No HOMO-LUMO gap: the purification gives up and the eigensolver forms the
    density, iteration by iteration as with eigensolver = householder."""
    mol = _degenerate(waters)
    out = []
    for solver in ("auto", "householder"):
        es = M.ElectronicStructure("mndo", M.SCFParams(max_iter=4, eigensolver=solver), context=ctx)
        es.SetMolecule(mol)
        try:
            es.DoSCF(True)
        except M.SCFNotConverged:
            pass
        out.append((es.GetIterations(), es.GetElectronicEnergy(), [t[1] for t in es.GetTrace()]))
    assert out[0][0] == out[1][0]
    # the guess has no gap at all: the first density is the eigensolver's own on both sides
    assert abs(out[0][2][0] - out[1][2][0]) <= 1e-12
    assert abs(out[0][1] - out[1][1]) <= 1e-8


def test_mixed_batch_of_gapped_and_degenerate(ctx):
    """A molecule's result does not depend on a neighbour that waits for the eigensolver."""
    prm = M.SCFParams(max_iter=60, damping_weight=0.0, diis_start_error=0.1, diis_end_error=0.0)
    good = W.water_cluster_k(4, 3)
    alone, q0 = M.batch_scf("mndo", [good, good], prm, context=ctx)
    both, q1 = M.batch_scf("mndo", [good, _degenerate(3)], prm, context=ctx)
    assert alone[0]["status"] == M.STATUS_CONVERGED
    assert both[0]["energy"] == alone[0]["energy"] and both[0]["iterations"] == alone[0]["iterations"]
    assert np.array_equal(q0[0], q1[0])


@pytest.mark.parametrize("waters", [22, 32, 33, 64])
def test_narrow_and_wide_tiles_agree(ctx, waters):
    """Alone a molecule's 128 x 32 tiles find an SM each; 60 of them take 128 x 64
    tiles.  Bases just above a row tile, at and beside a multiple of both widths, and
    of three row tiles."""
    mols = W.water_replicas(W.water_cluster_k(waters, 2), 60)
    prm = M.SCFParams(damping_weight=0.0, diis_start_error=0.1, diis_end_error=0.0)
    res, q = M.batch_scf("am1", mols, prm, context=ctx)
    for i in (0, 59):
        alone, qa = M.batch_scf("am1", [mols[i]], prm, context=ctx)
        assert alone[0]["iterations"] == res[i]["iterations"]
        assert alone[0]["energy"] == res[i]["energy"]
        assert np.array_equal(qa[0], q[i])
