"""GPU: the RVEA partition of many points, whose warps read the directions
themselves, equals the partition of the same points a few at a time, whose blocks
stage them (angles and indices bit for bit), on both sides of the lines."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,n,K", [(1, 4097, 3), (2, 4096, 600), (2, 4097, 600), (3, 16383, 100), (3, 16384, 100),
                                   (3, 16389, 513), (3, 16384, 8193), (5, 40959, 129), (5, 40960, 129), (8, 40961, 1000),
                                   (10, 16385, 128), (16, 16387, 31), (16, 16384, 700)])
def test_partition_of_many_points_equals_partition_of_few(M, n, K):
    from cuda_moea import stages as st
    g = torch.Generator(device="cuda").manual_seed(n + K)
    t = torch.rand((M, n), generator=g, device="cuda").clamp_min(1e-32)
    t[:, 5] = 1e-32
    t[:, 7] = t[:, 6]
    r = torch.rand((M, K), generator=g, device="cuda") + 0.01
    r /= r.norm(dim=0)
    r[:, K // 2] = r[:, 0]              # ties go to the smaller index
    ws = st.Workspace(n, M, K)
    theta, idx = st.rvea_partition(ws, t, r, 0, 0)
    for a in range(0, n, 4000):
        part = t[:, a:a + 4000].contiguous()
        th, ix = st.rvea_partition(ws, part, r, 0, 0)
        np.testing.assert_array_equal(ix.cpu().numpy(), idx[a:a + 4000].cpu().numpy())
        np.testing.assert_array_equal(th.view(torch.int32).cpu().numpy(), theta[a:a + 4000].view(torch.int32).cpu().numpy())
