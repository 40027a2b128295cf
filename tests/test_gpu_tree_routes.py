"""GPU: the paths that only direction sets on the far side of the dispatch lines
take: the cone tree (above 8,192 directions of four and five objectives, many
directions beside few points up to three), its batched form, and the batched niche
selection by sorts (fronts that a few directions hold)."""
import numpy as np
import pytest
import torch

import cuda_moea as cm

pytestmark = pytest.mark.gpu


def _directions(kind, M, H, rng):
    d = rng.standard_normal((M, H)) if kind == "signed" else np.abs(rng.standard_normal((M, H))) + 1e-3
    d /= np.linalg.norm(d, axis=0)
    if kind == "repeated":
        d = np.tile(d[:, :H // 4], 4)[:, rng.permutation(4 * (H // 4))]
    if kind == "nearly":     # a deviation that widens the margin: 5e-4 in length
        d *= 1.0 + rng.uniform(-4.9e-4, 4.9e-4, d.shape[1])
    return np.ascontiguousarray(d, np.float32)


@pytest.mark.parametrize("kind", ["positive", "signed", "repeated", "nearly"])
@pytest.mark.parametrize("M,n,H", [(1, 200, 40), (2, 300, 2000), (3, 700, 4000), (4, 500, 8200), (5, 600, 9000),
                                   (5, 60, 20000)])
def test_tree_matches_oracle(oracle, kind, M, n, H):
    from cuda_moea import stages as st
    rng = np.random.default_rng(H + n)
    d = _directions(kind, M, H, rng)
    x = rng.standard_normal((M, n)) if kind == "signed" else rng.random((M, n)) * rng.random(n) * 2
    x = x.astype(np.float32)
    x[:, :8] = d[:, :8] * 1.5
    x[:, 10] = 0.0
    x[:, 11] = 1e-30
    x[:, 12] = 3e18          # the squared length is finite, its margin wide
    x[:, 13] = 3e19          # the squared length overflows: every direction is a candidate
    x[M - 1, 14] = np.nan
    x[0, 15] = np.inf
    want_i, want_d = oracle.associate(x, d)
    got_i, got_d = st.associate(st.Workspace(n, M, d.shape[1]), torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda(),
                                st.ASSOC_TREE)
    np.testing.assert_array_equal(got_i.cpu().numpy(), want_i)
    np.testing.assert_array_equal(got_d.cpu().numpy(), want_d)


def _make(N, M, T, values, normalize=True, mode=0, kind="DTLZ2"):
    return cm.NSGA3(population_size=N, max_generations=T, problem=getattr(cm, kind)(M + 9, M), seed=N + M, print_progress=False,
                    reference_directions=cm.UserDefinedDirections(torch.from_numpy(values), normalize=normalize),
                    environment_selector=cm.NSGA3EnvironmentSelector(association_mode=mode))


def _same_as_alone(sizes, M, T, values, normalize=True):
    """A batch against the same instances alone, which visit every direction."""
    batch = cm.Batch([_make(N, M, T, values, normalize) for N in sizes])
    assert batch.fused
    batch.run()
    for i, N in enumerate(sizes):
        want, got = _make(N, M, T, values, normalize, mode=1).run(), batch.result(i)
        assert torch.equal(got.variables.view(torch.int32), want.variables.view(torch.int32))
        assert torch.equal(got.objectives.contiguous().view(torch.int32), want.objectives.contiguous().view(torch.int32))


@pytest.mark.parametrize("M,H", [(1, 40), (2, 2049), (3, 8193), (4, 8200), (5, 9000)])
def test_batched_tree_equals_every_direction_visited(M, H):
    values = _directions("positive", M, H, np.random.default_rng(H)).T.copy()
    _same_as_alone((92, 40, 300), M, 5, values)


@pytest.mark.parametrize("M,H", [(2, 300), (3, 9000), (8, 500)])
def test_batched_directions_of_any_length(M, H):
    values = (np.random.default_rng(H).random((H, M)) * 3 + 0.01).astype(np.float32)
    _same_as_alone((92, 40, 300), M, 5, values, normalize=False)


@pytest.mark.parametrize("M,H,sizes,T", [(3, 1, (1100, 92), 30), (3, 2, (2400,), 25), (2, 3, (3400, 1024), 20)])
def test_batched_niche_selection_by_sorts(M, H, sizes, T):
    """One to three directions: niche levels above those told apart, and buckets
    above those ranked by counting, in fronts shorter and longer than a block."""
    values = _directions("positive", M, H, np.random.default_rng(H)).T.copy()
    _same_as_alone(sizes, M, T, values)
