"""GPU: the non-dominated sort's tiles and rank merges at their edges against
the oracle: sizes around a tile, a merge group and both, with equal keys across
tile boundaries, runs of identical vectors, long runs of equal keys that are
not identical, and every class of violation."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _population(n, kind, rng):
    f = rng.random((3, n))
    if kind == "ties":            # few values: equal keys in every tile, identical vectors
        f = rng.integers(0, 4, (3, n)).astype(np.float64)
    elif kind == "long_runs":     # f0 and f1 + f2 constant on most points: one long run to order
        f[0] = 0.25
        f[1] = rng.integers(0, 1 << 12, n) / float(1 << 12)
        f[2] = 1.0 - f[1]
        f[:, ::7] = rng.random((3, len(f[0, ::7]))) + 1.0
    return f.astype(np.float32)


@pytest.mark.parametrize("kind", ["uniform", "ties", "long_runs"])
@pytest.mark.parametrize("n", [1, 2, 31, 1023, 1024, 1025, 2049, 8191, 8192, 8193, 9217, 16385, 66000])
def test_sort_edges_match_oracle(n, kind):
    from cuda_moea import stages as st
    from oracle import oracle as O
    rng = np.random.default_rng(n)
    objs = _population(n, kind, rng)
    cv = np.zeros(n, np.float32)
    if n % 2:                     # classes 1, 2 and 3 beside the feasible points
        pick = rng.random(n)
        cv = np.where(pick < 0.3, rng.integers(1, 5, n) / 4.0, 0.0).astype(np.float32)
        cv[pick > 0.98] = np.nan
        objs[1, (pick > 0.5) & (pick < 0.52)] = np.nan
    ws = st.Workspace(max(2, n), 3, 1)
    for target in (n, max(1, n // 2)):
        if kind == "uniform" and n > 20000 and target == n:
            continue              # hundreds of fronts on the host
        want, want_last = O.ndsort(cv, objs, target)
        got, got_last = st.ndsort(ws, torch.from_numpy(cv).cuda(), torch.from_numpy(objs).cuda(), target)
        np.testing.assert_array_equal(got.cpu().numpy(), want)
        assert got_last == want_last
