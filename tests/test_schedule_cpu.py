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
