"""Which kernel formed the density: the molecules of test_gpu_purify.py with a gap are
served by the purification itself, those without one (or with one too small) wait for
the eigensolver."""
import pytest

from engine_program import build_engine_program, run_engine_program, write_molecule
from test_gpu_purify import _degenerate, _molecule

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    return build_engine_program(tmp_path_factory.mktemp("engine"))


# 512 and 514, 544: a whole K segment, and the first sizes with a second one
@pytest.mark.parametrize("n", [2, 16, 18, 62, 64, 66, 80, 82, 112, 128, 130, 160, 162, 192, 194, 256, 258, 384, 510, 512,
                               514, 544, 546, 1024, 1026, 1030])
def test_gapped_molecule_is_purified(exe, tmp_path, n):
    r = run_engine_program(exe, "guess", write_molecule(tmp_path, 1, _molecule(n, n)))
    assert r.stdout == f"n {n} flags 0 iter 1 error 0\n", (r.stdout, r.stderr)


# The guess of an oxygen atom (beside water clusters): the atom alone has no gap.  With
# waters a lone pair of theirs is the LUMO instead, 5.5e-4, 1.6e-4 and 1.1e-3 above the
# atom's p level (oracle): 1.6e-4, 5e-5 and 3e-4 of the spectrum, which the one-CTA
# kernel's steps resolve and the tile kernel's 56 (25 waters) do not.
@pytest.mark.parametrize("waters,flag", [(0, 1), (3, 0), (15, 0), (25, 1)])
def test_small_gaps(exe, tmp_path, waters, flag):
    r = run_engine_program(exe, "guess", write_molecule(tmp_path, 0, _degenerate(waters)))
    assert r.stdout == f"n {6 * waters + 4} flags {flag} iter {1 - flag} error 0\n", (r.stdout, r.stderr)


@pytest.mark.parametrize("waters", [8, 32])
def test_executed_flops_count_the_steps(waters):
    """kernel_times()'s work: 34 digit products a step over 128-row tiles, by the steps taken."""
    import molds_gb300 as M
    from molds_gb300 import workloads as W
    ctx = M.Context(0)
    b = M.ResidentBatch("am1", [W.water_cluster_k(waters, 3)], context=ctx)
    p = M.SCFParams(damping_weight=0.0, diis_start_error=0.1, diis_end_error=0.0)
    b.run(p)
    b.profile(True)
    b.run(p)
    work = b.kernel_times()["purification"]["work"]
    iterations = b.results()[0][0]["iterations"]
    b.close()
    ctx.close()
    n = 6 * waters
    if n <= 128:
        step = 34 * 2 * 128 * 48 * 48
    else:                                   # 192: row tiles 0 (192 columns) and 1 (64 columns)
        step = 34 * 2 * 128 * (192 + 64) * 192
    steps = work / step
    assert steps == int(steps) and 12 * iterations <= steps <= 56 * iterations
