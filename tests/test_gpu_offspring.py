"""GPU: the offspring of a generation in one launch against the separate
mating, variation and evaluation kernels (reached through a mating callback
that returns the same parents), the crossover of long rows and the initial
population at the edges of their rules.  All comparisons are of bits, except
the host oracle's powf (the tolerance of the shorter rows)."""
import numpy as np
import pytest
import torch

import cuda_moea as cm
from cuda_moea import stages as st

import draws

pytestmark = pytest.mark.gpu


def _bits(t):
    return t.contiguous().view(torch.int32)


class SameParents(cm.PythonMating):
    """The library's own draws: tournament or the first candidate."""

    def __init__(self, seed, tournament):
        self.seed, self.tournament = seed, tournament

    def select(self, parents, state, context):
        n = parents["variables"].shape[0]
        cand = draws.mating_candidates(st, self.seed, context["generation"], n, state["active_count"])
        if not self.tournament:
            return cand[:, 0]
        return st.tournament(cand.contiguous(), state["rank"].contiguous(), parents["constraints"].contiguous())


def _compare(oracle, cls, problem, N, D, T=3, tournament=True, **kw):
    seed = 41
    own = cm.TournamentMating() if tournament else cm.RandomMating()
    runs = []
    for mating in (own, SameParents(oracle.derive_seed(seed), tournament)):
        a = cls(population_size=N, max_generations=T, problem=problem, seed=seed, mating=mating,
                print_progress=False, **kw)
        r = a.run()
        runs.append((r.variables.clone(), r.objectives.clone(), r.constraints.clone()))
    for x, y in zip(*runs):
        assert torch.equal(_bits(x), _bits(y))


@pytest.mark.parametrize("D", [3, 4, 5, 31, 32, 33, 64, 184, 185, 258, 259])
@pytest.mark.parametrize("N", [4, 6, 130])
def test_offspring_lengths(oracle, N, D):
    _compare(oracle, cm.NSGA3, cm.DTLZ2(D, 3), N, D)


@pytest.mark.parametrize("D", [32, 33, 184, 185])
@pytest.mark.parametrize("N", [16382, 16384])
def test_offspring_many_pairs(oracle, N, D):
    _compare(oracle, cm.NSGA3, cm.DTLZ1(D, 3), N, D, T=1)


@pytest.mark.parametrize("kind", ["DTLZ1", "DTLZ2", "DTLZ3", "DTLZ4", "DTLZ5", "DTLZ6", "DTLZ7", "ConvexDTLZ2",
                                  "C1DTLZ1", "C1DTLZ3", "C2DTLZ2", "C2ConvexDTLZ2", "C3DTLZ1", "C3DTLZ4"])
@pytest.mark.parametrize("D,M", [(12, 3), (41, 8)])
def test_offspring_problems(oracle, kind, D, M):
    _compare(oracle, cm.NSGA3, getattr(cm, kind)(D, M), 100, D, crossover=cm.SBX(20.0, 30.0, 0.9, 0.3),
             mutation=cm.PolynomialMutation(10.0, 20.0, 1.0))


@pytest.mark.parametrize("N", [3, 5, 101, 256])
def test_offspring_odd_populations_and_options(oracle, N):
    for mutation in (cm.PolynomialMutation(20.0, 20.0, 1.0), cm.NoMutation()):
        _compare(oracle, cm.RVEA, cm.DTLZ2(13, 3), N, 13, tournament=False, mutation=mutation)


@pytest.mark.parametrize("D", [703, 704, 705])
def test_offspring_rows_of_callback_problems(oracle, D):
    class Sum(cm.PythonProblem):
        def evaluate(self, x, context):
            f = x[:, 0] * 1.0
            return torch.stack((f, 1.0 - f), 1)

    _compare(oracle, cm.NSGA3, Sum(D, 2), 64, D)


@pytest.mark.parametrize("D", [1020, 1023, 1024, 1028, 2052])
@pytest.mark.parametrize("n", [2, 63, 64])
@pytest.mark.parametrize("sbx_prob,copy_prob", [(1.0, 0.0), (0.8, 0.4)])
def test_long_row_crossover(oracle, D, n, sbx_prob, copy_prob):
    """Aligned rows (the long-row kernel from 1024 variables) against the same
    rows at an address that keeps the general kernel, and the oracle."""
    rng = np.random.default_rng(D + n)
    parents = rng.random((n, D)).astype(np.float32)
    shifted = torch.empty(n * D + 1, device="cuda")[1:].view(n, D)
    aligned = torch.from_numpy(parents).cuda()
    shifted.copy_(aligned)
    bounds = torch.tile(torch.tensor([0.0, 1.0]), (D,)).cuda()
    cv, rank = torch.zeros(n, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    kw = dict(seed=7, generation=2, sbx_prob=sbx_prob, sbx_copy_prob=copy_prob)
    got, pidx = st.reproduce(aligned, cv, rank, n, bounds, n, **kw)
    general, pidx2 = st.reproduce(shifted, cv, rank, n, bounds, n, **kw)
    assert torch.equal(pidx, pidx2)
    assert torch.equal(_bits(got), _bits(general))
    u, sign, copy = draws.crossover_draws_np(oracle, 7, 2, n, D, sbx_prob, copy_prob)
    want = oracle.sbx(parents, pidx.cpu().numpy(), bounds.cpu().numpy(), u, sign, copy, 30.0, sbx_prob, copy_prob, n)
    want = oracle.pm(want, bounds.cpu().numpy(), draws.mutation_draws_np(oracle, 7, 2, n, D, 1.0), 20.0, 1.0)
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=5e-6, atol=5e-7)


@pytest.mark.parametrize("D", [4, 5, 7, 12, 1023, 1024])
@pytest.mark.parametrize("N", [4, 66])
def test_initial_population_draws(oracle, N, D):
    """Unit bounds: the draw itself, one Philox word per variable."""
    seed = 99
    a = cm.NSGA3(population_size=N, max_generations=1, problem=cm.DTLZ2(D, 3), seed=seed, print_progress=False)
    a.initialize()
    w = oracle.philox_stream(oracle.derive_seed(seed), 0, 1, (N * D + 3) // 4).reshape(-1)[: N * D]
    want = ((w >> 8).astype(np.float32) * np.float32(2.0 ** -24)).reshape(N, D)
    np.testing.assert_array_equal(a.population.variables.cpu().numpy(), want)
