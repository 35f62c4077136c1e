"""The core Hamiltonian's kernels leave the pair energies as they are."""
import pytest

from engine_program import build_engine_program, run_engine_program, write_molecule
from molds_gb300 import workloads as W

pytestmark = pytest.mark.gpu


# one row of pairs, rows beyond a warp, and a basis whose atoms fill several CTAs
@pytest.mark.parametrize("waters", [1, 14, 40])
def test_core_energy_twice(tmp_path, waters):
    exe = build_engine_program(tmp_path)
    r = run_engine_program(exe, "hcore", write_molecule(tmp_path, 1, W.water_cluster_k(waters, 3)))
    assert r.returncode == 0, (r.stdout, r.stderr)
    first, again = r.stdout.splitlines()
    assert first == again
