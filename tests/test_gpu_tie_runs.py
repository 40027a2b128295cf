"""GPU: runs of equal sort keys (the same f0 and the same sum of the others) of
every length around the one that is ranked member by member, with different and
with identical vectors in them, against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [3, 5, 16])
@pytest.mark.parametrize("length", [2, 3, 31, 32, 33, 34, 65])
@pytest.mark.parametrize("values", [2, 4096])  # few: identical vectors; many: different ones
def test_runs_of_equal_keys(M, length, values):
    from cuda_moea import stages as st
    from oracle import oracle as O
    rng = np.random.default_rng(1000 * M + length + values)
    n = 1400
    run = np.arange(n) // length
    f = np.empty((M, n))
    f[0] = (run * 37 % 101) / 128.0
    f[1:M - 1] = rng.integers(0, values, (M - 2, n)) / 4096.0
    f[M - 1] = (M - 2) - f[1:M - 1].sum(0) + run % 3   # exact sums: the same S through a run
    f = np.ascontiguousarray(f[:, rng.permutation(n)], np.float32)
    cv = np.zeros(n, np.float32)
    want, want_last = O.ndsort(cv, f, n)
    got, got_last = st.ndsort(st.Workspace(n, M, 1), torch.from_numpy(cv).cuda(), torch.from_numpy(f).cuda(), n)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    assert got_last == want_last
