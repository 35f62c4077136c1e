"""A wait of the purification for a copy or an MMA that runs out: the kernels
return, the molecule is left to the eigensolver, the host is told.  The limit is
set to zero, so that every wait runs out before what it waits for has come; the
kernels then wait for it with their usual limit before they go on."""
import pytest

from engine_program import build_engine_program, run_engine_program, write_molecule
from molds_gb300 import workloads as W

pytestmark = pytest.mark.gpu

AM1 = 1


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    return build_engine_program(tmp_path_factory.mktemp("engine"))


# 12 (one group of levels), 78 (three), 126 (four), 132 and 546 basis functions (tiles; two K segments)
@pytest.mark.parametrize("waters", [2, 13, 21, 22, 91])
def test_wait_that_runs_out(exe, tmp_path, waters):
    r = run_engine_program(exe, "waits", write_molecule(tmp_path, AM1, W.water_cluster_k(waters, 3)))
    assert r.returncode == 0, (r.stdout, r.stderr)
    lines = r.stdout.splitlines()
    # flagged for the eigensolver, not advanced, error set; then as if nothing had happened
    assert lines[0] == "pass 0 flags 1 iter 0 error 1"
    assert lines[1] == "pass 1 flags 0 iter 1 error 0"
    assert lines[2] == "same_density 1"
    # an SCF whose waits run out is right (the eigensolver's densities) and reports them once
    assert lines[3].startswith("scf_error tensor cores: a wait")
    assert lines[5] == "scf_ok 1" and lines[7] == "scf_ok 1"
    limited, after, plain = (lines[k].split() for k in (4, 6, 8))
    assert limited[3] == plain[3] in ("1", "2")   # 91 waters do not converge within 60 iterations, nor does the oracle
    assert after == plain
    assert limited[5] == plain[5]
    assert abs(float(limited[1]) - float(plain[1])) <= 1e-9


def test_server_reports_a_wait_that_ran_out(exe, tmp_path):
    r = run_engine_program(exe, "server", write_molecule(tmp_path, AM1, W.water_cluster_k(2, 3)))
    assert r.returncode == 0, (r.stdout, r.stderr)
    lines = r.stdout.splitlines()
    assert lines[0].startswith("served status 1")
    assert len(lines) == 2 and lines[1].startswith("poll_error server stopped: lane 0: tensor cores: a wait")
