"""GPU: the dense association at its edges against the oracle (indices and
distances bit for bit): 32- and 64-point CTAs and their remainders, direction
counts around a chunk of 32 and around the tile count (tiles of one, two and
more chunks), repeated directions (ties), zero, non-finite and far points,
directions that are not of unit length."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 10, 16])
@pytest.mark.parametrize("n,H", [(1, 1), (31, 33), (33, 32), (65, 4097), (130, 8193), (9472, 65), (9473, 127),
                                 (9535, 2)])
def test_dense_search_matches_oracle(M, n, H):
    from cuda_moea import stages as st
    from oracle import oracle as O
    rng = np.random.default_rng(100 * n + H + M)
    x = rng.random((M, n)).astype(np.float32)
    x[:, ::17] = 0.0
    if n > 40:
        x[0, 3] = np.inf
        x[M - 1, 5] = np.nan
        x[:, 7] = 1e18
        x[:, 9] = 1e-22
    d = rng.random((M, H)) + 1e-3
    d /= np.linalg.norm(d, axis=0)
    if H > 4:
        d[:, H // 2] = d[:, 1]
        d[:, H - 1] = d[:, 1]
    if H == 127:
        d *= 1.01                       # re-scored against every direction
    d = d.astype(np.float32)
    ws = st.Workspace(max(n, 2), M, H)
    want_i, want_d = O.associate(x, d)
    got_i, got_d = st.associate(ws, torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda(), st.ASSOC_SCAN)
    np.testing.assert_array_equal(got_i.cpu().numpy(), want_i)
    np.testing.assert_array_equal(got_d.cpu().numpy(), want_d)
