"""GPU: sorts whose first fronts are thin, which one CTA finishes, and their
neighbours (the sizes around its lines, fronts that widen later, infeasible
points behind the fronts, repeated points), against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _objectives(kind, M, n, rng):
    f = np.empty((M, n))
    t = rng.permutation(n) / 1024.0
    if kind == "chain":              # every point its own front
        f[:] = t
    elif kind == "pairs":            # two points a front, M > 1
        f[:] = np.floor(t * 512) / 512
        f[0, ::2] += 1.0 / 4096
        f[-1, 1::2] += 1.0 / 4096
    elif kind == "repeated":         # runs of identical points, one front each
        f[:] = np.floor(t * 128) / 128
    elif kind == "widening":         # a chain of twelve points before one wide front
        x = rng.random(n)
        f[:] = 1.0
        f[0], f[-1] = 1.0 + x, 2.0 - x
        f[:, :12] = np.arange(12) / 32.0
    return f.astype(np.float32)


@pytest.mark.parametrize("kind", ["chain", "pairs", "repeated", "widening"])
@pytest.mark.parametrize("M,n", [(1, 600), (2, 520), (2, 1025), (2, 2048), (2, 2049), (3, 1500), (2, 4097), (2, 8192),
                                 (2, 8193), (3, 8191)])
@pytest.mark.parametrize("infeasible", [False, True])
def test_thin_fronts_match_oracle(kind, M, n, infeasible):
    from cuda_moea import stages as st
    from oracle import oracle as O
    rng = np.random.default_rng(n + M)
    f = _objectives(kind, M, n, rng)
    cv = np.zeros(n, np.float32)
    if infeasible:
        pick = rng.random(n)
        cv = np.where(pick < 0.6, rng.integers(1, 9, n) / 8.0, 0.0).astype(np.float32)
        cv[pick > 0.99] = np.nan
        f[0, (pick > 0.7) & (pick < 0.71)] = np.nan
    ws = st.Workspace(n, M, 1)
    for target in (n, n // 2, 1):
        want, want_last = O.ndsort(cv, f, target)
        got, got_last = st.ndsort(ws, torch.from_numpy(cv).cuda(), torch.from_numpy(f).cuda(), target)
        np.testing.assert_array_equal(got.cpu().numpy(), want)
        assert got_last == want_last
