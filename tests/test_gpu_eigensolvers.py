"""The eigensolvers that the default path does not take: precision = mixed with the
Householder path (FP32 back-transformation, density on the tensor cores in 3xTF32, then
the FP64 phase) and the Jacobi eigensolvers, against the oracle."""
import numpy as np
import pytest

import molds_gb300 as M
from molds_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SCF = dict(max_iter=500, rms_density=1e-8, damping_thresh=1.0, damping_weight=0.0, diis_num_error_vect=5,
           diis_start_error=0.1, diis_end_error=0.0)
E_TOL = {"fp64": 1e-8, "mixed": 1e-6}
Q_TOL = 1e-6


@pytest.fixture(scope="module")
def ctx():
    c = M.Context(0)
    yield c
    c.close()


_refs = {}


def _ref(theory, waters):
    if (theory, waters) not in _refs:
        mol = W.water_cluster_k(waters, 3)
        _refs[theory, waters] = mol, O.scf(O.make_molecule(theory, mol.Z, mol.xyz), O.SCFParams(**SCF))
    return _refs[theory, waters]


# 12; 48 and 96: shared memory; 216: above 194 (the block Jacobi, the cluster tridiagonalisation)
CASES = [("mixed", "householder", w) for w in (2, 8, 16, 36)] + [("fp64", "jacobi", w) for w in (2, 8, 16, 36)] + \
        [("mixed", "jacobi", w) for w in (2, 16)]


@pytest.mark.parametrize("precision,solver,waters", CASES)
def test_single_molecule(ctx, precision, solver, waters):
    mol, ref = _ref("am1", waters)
    es = M.ElectronicStructure("am1", M.SCFParams(**SCF, precision=precision, eigensolver=solver), context=ctx)
    es.SetMolecule(mol)
    es.DoSCF(True)
    assert abs(es.GetElectronicEnergy(0) - ref.energy) < E_TOL[precision]
    assert np.max(np.abs(es.GetMullikenCharges() - ref.charges)) < Q_TOL
    if precision == "fp64":
        assert es.GetIterations() == ref.iterations


@pytest.mark.parametrize("precision,solver", [("mixed", "householder"), ("fp64", "jacobi"), ("mixed", "jacobi")])
def test_batch(ctx, precision, solver):
    """Twelve molecules of three sizes: more than the cluster Jacobi takes."""
    waters = [2, 8, 16] * 4
    refs = [_ref("am1", w) for w in waters]
    res, q = M.batch_scf("am1", [m for m, _ in refs], M.SCFParams(**SCF, precision=precision, eigensolver=solver),
                         context=ctx)
    for r, qi, (_, ref) in zip(res, q, refs):
        assert r["status"] == M.STATUS_CONVERGED
        assert abs(r["energy"] - ref.energy) < E_TOL[precision]
        assert np.max(np.abs(qi - ref.charges)) < Q_TOL
