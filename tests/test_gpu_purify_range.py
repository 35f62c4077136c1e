"""Digit sums of the purification of dense matrices stay in the range that their
recombination covers, so the eigensolver is not needed for them."""
import numpy as np
import pytest

from engine_program import build_engine_program, run_engine_program

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    return build_engine_program(tmp_path_factory.mktemp("engine"))


def purify(exe, directory, F, nocc):
    """flags, error word and P of launch_purify_small / launch_purify_big for one matrix"""
    n = F.shape[0]
    with open(directory / "in.bin", "wb") as f:
        f.write(np.array([n, nocc], dtype=np.int32).tobytes() + np.ascontiguousarray(F).tobytes())
    r = run_engine_program(exe, "purify", directory / "in.bin", directory / "out.bin")
    assert r.returncode == 0, (r.stdout, r.stderr)
    raw = open(directory / "out.bin", "rb").read()
    flags, err = np.frombuffer(raw[:8], dtype=np.int32)
    return int(flags), int(err), np.frombuffer(raw[8:]).reshape(n, n)


# one K segment (512), two with a remainder, and four with one: sums over whole
# segments of a dense matrix have a mean of 0.67 * 2^22 on the diagonal and spread
# by 0.09 * 2^22, so at n = 2064 some of 24 steps' 10^5 of them pass 2^22
@pytest.mark.parametrize("n,seed", [(128, 0), (130, 0), (512, 0), (514, 0), (544, 0), (1032, 2), (2064, 0), (2064, 1)])
def test_dense_matrix_is_purified(exe, tmp_path, n, seed):
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.normal(size=(n, n)))
    w = np.sort(rng.uniform(0.3, 1.0, n))
    nocc = n // 3
    w[:nocc] *= -1.0
    F = (q * w) @ q.T
    F = 0.5 * (F + F.T)
    flags, err, P = purify(exe, tmp_path, F, nocc)
    assert err == 0
    assert flags == 0
    v = np.linalg.eigh(F)[1][:, :nocc]
    # numpy's projector is off by about n eps ||F|| / gap; five times that
    assert np.abs(P - 2.0 * v @ v.T).max() <= 5 * n * 2.2e-16 / 0.6
    assert np.array_equal(P, P.T)
