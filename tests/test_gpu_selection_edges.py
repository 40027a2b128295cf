"""GPU: the selections at the sizes where their launches change: the merged
points around the limits of the cluster launch that extracts, translates and
solves the intercepts, and around the size up to which a point's translation
is taken inside the RVEA partition."""
import numpy as np
import pytest
import torch

import cuda_moea as cm
from cuda_moea import stages as st

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [2, 3, 10])
@pytest.mark.parametrize("N", [1, 2, 255, 256, 257, 4095, 4096, 4097, 16383, 16384, 16385])
def test_nsga3_selection_around_the_cluster_limits(oracle, M, N):
    rng = np.random.default_rng(N + M)
    objs = rng.random((M, 2 * N)).astype(np.float32)
    cv = np.where(rng.random(2 * N) < 0.1, rng.random(2 * N), 0).astype(np.float32)
    refs = oracle.reference_directions(0, min(N, 300) + 1, M)
    ideal = objs[:, :N].min(1).astype(np.float32)
    ws = st.Workspace(2 * N, M, refs.shape[1])
    want = oracle.nsga3_select(cv, objs, refs, 12345, 9, ideal)
    got = st.nsga3_select(ws, torch.from_numpy(cv).cuda(), torch.from_numpy(objs).cuda(),
                          torch.from_numpy(refs).cuda(), 12345, 9, torch.from_numpy(ideal).cuda())
    for key in ("sizes", "survivors", "fronts", "ideal"):
        np.testing.assert_array_equal(got[key].cpu().numpy(), want[key])
    assert got["offset"] == want["offset"]


@pytest.mark.parametrize("N,M", [(64, 3), (1023, 8), (1024, 8), (1025, 8), (2047, 4), (2048, 4), (2049, 4)])
def test_rvea_generations_equal_the_stage_calls(oracle, N, M):
    """Every generation of a handle against the stage calls on the same
    offspring: survivors, objectives and the active count, bit for bit."""
    D, T, seed, alpha = 14, 12, 5, 2.0
    algo = cm.RVEA(population_size=N, max_generations=T, problem=cm.DTLZ2(D, M), seed=seed,
                   reference_directions=cm.AdaptiveRVEADirections(frequency=1.0), print_progress=False)
    algo.initialize()
    refs = algo.reference_directions.clone().contiguous()
    K = refs.shape[1]
    pop = algo.population
    x, f, cv, active = pop.variables.clone(), pop.objectives.t().contiguous(), pop.constraints.clone(), N
    bounds = torch.tile(torch.tensor([0.0, 1.0]), (D,)).cuda()
    dseed = oracle.derive_seed(seed)
    ws = st.Workspace(2 * N, M, K)
    gamma = st.rvea_gamma(ws, refs)
    for g in range(4):
        ox, _ = st.reproduce(x, cv, None, active, bounds, N, mating=0, seed=dseed, generation=g)
        of, ocv = st.problem_evaluate(2, ox, M)
        mx, mf, mcv = torch.cat([x, ox]), torch.cat([f, of], 1), torch.cat([cv, ocv])
        t, _ = st.rvea_translate(ws, mf)
        theta, idx = st.rvea_partition(ws, t, refs, active, N)
        apd = st.rvea_apd(ws, t, theta, gamma, idx, g + 1, T, alpha)
        sel, act = st.rvea_elitism(ws, idx, mcv, apd, N, K)
        algo.step()
        r = algo.result()
        assert r.active_count == act
        s = sel.long()
        assert torch.equal(r.variables[:act], mx[s])
        assert torch.equal(r.objectives[:act], mf[:, s].t())
        nan = float("nan")
        x = torch.full_like(x, nan)
        f = torch.full_like(f, nan)
        cv = torch.full_like(cv, nan)
        x[:act], f[:, :act], cv[:act] = mx[s], mf[:, s], mcv[s]
        active = act


@pytest.mark.parametrize("kind,M", [("DTLZ4", 3), ("DTLZ1", 2), ("DTLZ7", 8)])
def test_batch_peel_of_thin_and_wide_fronts(kind, M):
    """Hundreds of thin fronts (short queues, a warp or eight lanes per row)
    and few wide ones (long queues, lists longer than one thread follows),
    against the same instances alone."""
    def make(N):
        return cm.NSGA3(population_size=N, max_generations=6, problem=getattr(cm, kind)(M + 19, M), seed=N,
                        print_progress=False)

    sizes = [46, 92, 130, 510, 512, 514, 2050, 4096]
    batch = cm.Batch([make(N) for N in sizes])
    assert batch.fused
    batch.run()
    for i, N in enumerate(sizes):
        want, got = make(N).run(), batch.result(i)
        assert torch.equal(got.variables, want.variables)
        assert torch.equal(got.objectives, want.objectives)
        assert torch.equal(got.auxiliary_indices, want.auxiliary_indices)


class _Spheres(cm.PythonProblem):
    def __init__(self):
        super().__init__(6, 2)

    def evaluate(self, x, context):
        return torch.stack((x.square().sum(1), (x - 1).square().sum(1)), 1)


def _callback_run(cls, graphs, seed=3):
    with torch.cuda.stream(torch.cuda.Stream()):
        algo = cls(population_size=64, max_generations=5, problem=_Spheres(), seed=seed, print_progress=False,
                   use_graphs=graphs)
        algo.initialize()
    torch.cuda.synchronize()
    return algo


@pytest.mark.parametrize("cls", [cm.NSGA3, cm.RVEA])
def test_callback_selection_graph_over_resets(cls):
    """The selection's graphs outlive a reset after an odd number of
    generations: every run equals the one of direct launches."""
    a, b = _callback_run(cls, True), _callback_run(cls, False)
    for _ in range(3):
        x, y = a.run(), b.run()
        assert torch.equal(x.variables.view(torch.int32), y.variables.view(torch.int32))
        assert torch.equal(x.objectives.contiguous().view(torch.int32), y.objectives.contiguous().view(torch.int32))
        a.reset()
        b.reset()


@pytest.mark.parametrize("cls", [cm.NSGA3, cm.RVEA])
def test_callback_generations_inside_the_callers_capture(cls):
    """A caller that captures the generations of a callback problem in a graph
    of its own gets the same populations."""
    a, b = _callback_run(cls, True), _callback_run(cls, True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=a.stream):
        a.step()
        a.step()
    graph.replay()
    torch.cuda.synchronize()
    for _ in range(2):
        b.step()
    x, y = a.result(), b.result()
    assert torch.equal(x.variables.view(torch.int32), y.variables.view(torch.int32))


@pytest.mark.parametrize("M", [1, 2, 3, 5, 10])
@pytest.mark.parametrize("n", [2, 600, 9500])
def test_dense_search_of_points_whose_distances_overflow(oracle, M, n):
    """A point all of whose distances are infinite has no direction (-1)."""
    rng = np.random.default_rng(n + M)
    x = (rng.random((M, n)) * 3e38).astype(np.float32)
    x[:, rng.random(n) < 0.2] = -0.0
    d = rng.random((M, 37)) + 0.01
    d = (d / np.linalg.norm(d, axis=0)).astype(np.float32)
    want_i, want_d = oracle.associate(x, d)
    got_i, got_d = st.associate(st.Workspace(n, M, 37), torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda(),
                                st.ASSOC_SCAN)
    np.testing.assert_array_equal(got_i.cpu().numpy(), want_i)
    np.testing.assert_array_equal(got_d.cpu().numpy(), want_d)
