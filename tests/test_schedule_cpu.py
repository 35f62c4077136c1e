"""The host rules that choose between launches (csrc/schedule.h)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("schedule") / "schedule_main")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "molds_gb300", "csrc"),
                    os.path.join(HERE, "cpp", "schedule_main.cpp"), "-o", exe], check=True)
    return lambda *a: subprocess.run([exe] + [str(x) for x in a], capture_output=True, text=True, check=True).stdout


# 18 clusters of eight CTAs fit 152 SMs
@pytest.mark.parametrize("count,n,pays", [
    (1, 194, 0), (1, 195, 1), (18, 195, 1), (19, 195, 0), (36, 234, 1), (37, 234, 0), (38, 300, 1), (54, 300, 1),
    (55, 300, 0),
    (152, 300, 0),   # four groups of 38: counted by group each would take three waves
    (64, 234, 0),    # four groups of 16
    (10000000, 400, 0)])
def test_cluster_rule(rule, count, n, pays):
    assert int(rule("cluster", count, n, 18)) == pays


def test_size_buckets(rule):
    edges = [31, 64, 96, 128, 160, 194, 256, 338]
    for k, e in enumerate(edges):
        assert int(rule("bucket", e)) == k and int(rule("bucket", e + 1)) == k + 1
    assert int(rule("bucket", 1)) == 0 and int(rule("bucket", 100000)) == len(edges)


NEVER = 1000   # steps that no iteration has


def _scf(rule, mols, tiled=1, block=3, max_iter=100, gapless=0):
    """iterations of each effort; (status, waits) of each molecule (converged, from, steps)"""
    out = [int(x) for x in rule("scf", tiled, 6, gapless, block, max_iter, 32, 56, *[v for m in mols for v in m]).split()]
    return out[:3], list(zip(out[3::2], out[4::2]))


@pytest.mark.parametrize("block", [1, 2, 3])
def test_effort_without_waits(rule, block):
    used, mols = _scf(rule, [(20, 0, 24), (31, 0, 32)], block=block)
    assert mols == [(1, 0), (1, 0)]
    assert used[1:] == [6, 0] and used[0] <= 25 + 2 * block


@pytest.mark.parametrize("block", [1, 2, 3])
@pytest.mark.parametrize("steps", [33, 56])
def test_more_steps_settle_without_the_eigensolver(rule, block, steps):
    """A molecule that goes on needing more than the few steps: it waits twice at
    most, once for each raise, and the eigensolver is never launched."""
    used, mols = _scf(rule, [(20, 0, 24), (60, 8, steps)], block=block)
    assert mols[0] == (1, 0) and mols[1][0] == 1
    assert used[2] == 0
    assert mols[1][1] <= 4 * block
    assert sum(used) <= 60 + 7 * block


@pytest.mark.parametrize("block", [1, 2, 3])
@pytest.mark.parametrize("tiled", [0, 1])
def test_no_gap_takes_the_eigensolver(rule, block, tiled):
    used, mols = _scf(rule, [(20, 0, 24), (40, 0, NEVER)], tiled=tiled, block=block)
    assert mols[0] == (1, 0) and mols[1][0] == 1
    assert used[2] >= 38 and mols[1][1] <= 4 * block
    assert sum(used) <= 40 + 7 * block


@pytest.mark.parametrize("block", [1, 2, 3])
@pytest.mark.parametrize("tiled", [0, 1])
def test_single_iteration_without_a_gap(rule, block, tiled):
    """One iteration that needs the eigensolver, and one later that needs all steps."""
    used, mols = _scf(rule, [(40, 12, 24), (41, 40, NEVER)], tiled=tiled, block=block)
    assert mols[0] == (1, 0) and mols[1][0] == 1 and used[2] >= 1


@pytest.mark.parametrize("max_iter", [1, 2, 7])
@pytest.mark.parametrize("mol", [(50, 0, 24), (50, 0, 40), (50, 0, NEVER), (50, 6, NEVER)])
def test_max_iter_ends_the_loop(rule, max_iter, mol):
    """Molecules that waited are carried past max_iter until they have had it."""
    used, mols = _scf(rule, [mol, (50, 0, 24)], max_iter=max_iter)
    assert [m[0] for m in mols] == [2, 2]


@pytest.mark.parametrize("block", [1, 2, 3])
@pytest.mark.parametrize("tiled", [0, 1])
def test_known_gapless_never_waits(rule, block, tiled):
    used, mols = _scf(rule, [(20, 0, 24), (2, 0, NEVER)], tiled=tiled, block=block, gapless=1)
    assert mols == [(1, 0), (1, 0)]
    assert used[:2] == [0, 0] and used[2] <= 20 + 2 * block
