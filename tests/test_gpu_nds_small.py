"""GPU: the one-CTA sort of small populations at its edges against the oracle
and against the general sort (forced through the workspace): sizes around a
word and up to its limit and one beyond, every class of violation, NaN and
infinite objectives, ties, every stop target that matters."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 16])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 184, 257, 511, 512, 513])
@pytest.mark.parametrize("kind", ["uniform", "ties", "mixed"])
def test_small_sort_matches_oracle_and_general(M, n, kind):
    from cuda_moea import stages as st
    from oracle import oracle as O
    rng = np.random.default_rng(31 * n + M)
    f = rng.random((M, n)) if kind != "ties" else rng.integers(0, 3, (M, n)).astype(np.float64)
    f = f.astype(np.float32)
    cv = np.zeros(n, np.float32)
    if kind == "mixed":
        pick = rng.random(n)
        cv = np.where(pick < 0.4, rng.integers(0, 6, n) / 5.0 - 0.2, 0.0).astype(np.float32)
        cv[pick > 0.95] = np.nan
        cv[(pick > 0.93) & (pick < 0.95)] = np.inf
        f[M - 1, (pick > 0.5) & (pick < 0.55)] = np.nan
        f[0, (pick > 0.55) & (pick < 0.6)] = np.inf
        f[0, (pick > 0.6) & (pick < 0.63)] = -0.0
    small, general = st.Workspace(max(n, 2), M, 1), st.Workspace(max(n, 2), M, 1)
    general.set_peel(True)
    for target in {n, max(1, n // 2), 1}:
        want, want_last = O.ndsort(cv, f, target)
        for ws in (small, general):
            got, got_last = st.ndsort(ws, torch.from_numpy(cv).cuda(), torch.from_numpy(f).cuda(), target)
            np.testing.assert_array_equal(got.cpu().numpy(), want)
            assert got_last == want_last
