"""A molecule's tridiagonalisation runs in a cluster of CTAs in a short list and in
one CTA in a long one; the two form the same sums in the same order."""
import numpy as np
import pytest

import molds_gb300 as M
from molds_gb300 import workloads as W


# 198: just above the smallest basis of the cluster kernel; 234, 306: rows that do
# not fill the last round of CTAs; 396: near the largest basis below the whole-GPU kernels
@pytest.mark.gpu
@pytest.mark.parametrize("waters", [33, 39, 51, 66])
def test_cluster_and_one_cta_agree(waters):
    mols = W.water_replicas(W.water_cluster_k(waters, seed=2), 90)
    p = M.SCFParams(precision="fp64", eigensolver="householder")
    ctx = M.Context(0)
    res, charges = M.batch_scf("am1", mols, p, context=ctx)
    for i in (0, 89):
        alone, q = M.batch_scf("am1", [mols[i]], p, context=ctx)
        assert alone[0]["iterations"] == res[i]["iterations"]
        assert alone[0]["energy"] == res[i]["energy"]
        assert np.array_equal(q[0], charges[i])
