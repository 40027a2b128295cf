"""GPU: the search over every direction on both sides of the lines between its
two forms (dense and split over ranges of directions), and with directions that
are not of unit length, against the oracle (indices and distances bit for bit)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(x, d, **spec):
    from cuda_moea import stages as st
    from oracle import oracle as O
    M, n = x.shape
    want_i, want_d = O.associate(x, d)
    X, D = torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda()
    ws = st.Workspace(max(n, 2), M, d.shape[1])
    for got_i, got_d in (st.associate(ws, X, D, st.ASSOC_SCAN), st.associate_static(X, D),
                         st.associate(ws, X, D, st.ASSOC_TREE)):
        np.testing.assert_array_equal(got_i.cpu().numpy(), want_i)
        np.testing.assert_array_equal(got_d.cpu().numpy(), want_d)


def _points(rng, M, n, d):
    x = (rng.random((M, n)) * rng.random(n) * 2).astype(np.float32)
    k = min(n, d.shape[1], 8)
    x[:, :k] = d[:, :k] * 1.5
    if n > 40:
        x[:, 16:20] = 0.0
        x[:, 20] = 1e-30
        x[:, 21] = 3e18
        x[M - 1, 22] = np.nan
        x[0, 23] = np.inf
        x[:, 24] = np.inf
        x[0, 25] = -np.inf
    return x


# (points, directions) beside the lines: 64 directions; 128 (64 from twelve
# objectives on) points per direction; 12,288 directions (8,192 from twelve objectives on) and six per point;
# 4,096 and 2,048 directions of two objectives
LINES = [(1, 1000, 700), (3, 70, 64), (3, 70, 65), (3, 8320, 65), (3, 8319, 65), (12, 4160, 65), (12, 4159, 65),
         (3, 100, 12288), (3, 100, 12289), (4, 2048, 12289), (4, 2049, 12289), (16, 90, 8192), (16, 90, 8193), (5, 33, 20000), (2, 300, 4096),
         (2, 300, 4097), (2, 9472, 2048), (2, 9472, 2049), (16, 64, 13000)]


@pytest.mark.parametrize("M,n,H", LINES)
def test_both_sides_of_the_lines(M, n, H):
    rng = np.random.default_rng(n + H + M)
    d = np.abs(rng.standard_normal((M, H))) + 1e-3
    d = (d / np.linalg.norm(d, axis=0)).astype(np.float32)
    d[:, H // 2] = d[:, 0]
    d[:, H - 1] = d[:, 0]
    _check(_points(rng, M, n, d), d)


@pytest.mark.parametrize("signs", [False, True])
@pytest.mark.parametrize("M,n,H", [(2, 33, 100), (3, 70, 33), (3, 31, 257), (5, 300, 1001), (8, 64, 4000), (8, 14209, 115),
                                   (3, 14300, 130), (10, 500, 700), (16, 65, 300), (16, 14208, 240), (4, 100, 13000)])
def test_directions_that_are_not_of_unit_length(M, n, H, signs):
    rng = np.random.default_rng(n + H + M)
    d = (rng.random((M, H)) * 3 + 0.01).astype(np.float32)
    if signs:
        d *= np.where(rng.random((M, H)) < 0.5, -1, 1).astype(np.float32)
        d[:, 3] = 0.0
        d[0, 5] = np.inf
        d[M - 1, 7] = np.nan
        d[:, 9] = 1e25
    d[:, H // 2] = d[:, 1]
    d[:, H - 1] = d[:, 1]
    x = _points(rng, M, n, np.where(np.isfinite(d), d, 1).astype(np.float32))
    _check(x, d)
