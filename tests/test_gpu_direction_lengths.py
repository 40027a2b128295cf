"""GPU: the largest deviation of a direction from unit length is found wherever
the direction lies among them.  A point on the longer direction J (length 1.0004)
is nearer to a unit direction K at an angle of 4e-4, although J has the larger
projection: K is found only when J's deviation widens the candidate margin."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [3, 6])
@pytest.mark.parametrize("H,J", [(2, 1), (40, 39), (513, 512), (4200, 5), (4200, 511), (4200, 516), (4200, 1100),
                                 (4200, 1600), (4200, 2050), (4200, 2999), (4200, 3100), (4200, 4095), (4200, 4101),
                                 (4200, 4199)])
def test_length_deviation_of_any_direction_counts(M, H, J):
    from cuda_moea import stages as st
    from oracle import oracle as O
    rng = np.random.default_rng(10 * H + J + M)
    d = np.abs(rng.standard_normal((M, H))) + 0.05
    d /= np.linalg.norm(d, axis=0)
    u = d[:, J].copy()
    side = rng.standard_normal(M)
    side -= side.dot(u) * u
    side /= np.linalg.norm(side)
    K = 0 if J else 1
    d[:, K] = np.cos(4e-4) * u + np.sin(4e-4) * side
    d[:, J] = 1.0004 * u
    d = d.astype(np.float32)
    n = 70
    x = (rng.random((M, n)) * 2).astype(np.float32)
    x[:, 3] = u
    x[:, 40] = 3.0 * u
    want_i, want_d = O.associate(x, d)
    assert want_i[3] == K and want_i[40] == K
    ws = st.Workspace(n, M, H)
    for mode in (st.ASSOC_TREE, st.ASSOC_SCAN, st.ASSOC_TENSOR):
        got_i, got_d = st.associate(ws, torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda(), mode)
        np.testing.assert_array_equal(got_i.cpu().numpy(), want_i, err_msg=f"mode {mode}")
        np.testing.assert_array_equal(got_d.cpu().numpy(), want_d, err_msg=f"mode {mode}")
