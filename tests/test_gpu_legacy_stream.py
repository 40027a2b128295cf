"""GPU: callback problems on the legacy default stream, which no graph can be
captured from: the generations are launched directly, with the same results."""
import ctypes

import pytest
import torch

import cuda_moea as cm
from cuda_moea import _lib
from cuda_moea._lib import check, lib

pytestmark = pytest.mark.gpu

LEGACY_STREAM = 1  # the handle cudaStreamLegacy


def _evaluate(user, x, f, cv, N, D, M, generation, generations, stream):
    return lib().moea_problem_evaluate(2, x, N, D, M, f, cv, stream)


def _run(cls, N, stream):
    """Objectives and variables after a run, a reset and another run of DTLZ2
    as the caller's own problem on `stream`, through the C interface."""
    cfg, keep = cls(population_size=N, max_generations=4, problem=cm.DTLZ2(12, 3), seed=5,
                    print_progress=False)._build_config()
    keep.append(_lib.EVALUATE_FN(_evaluate))
    cfg.problem_kind, cfg.evaluate, cfg.stream, cfg.use_graphs = 0, keep[-1], stream, 1
    handle, ms, out = ctypes.c_void_p(), ctypes.c_double(), []
    check(lib().moea_algorithm_create(ctypes.byref(cfg), ctypes.byref(handle)))
    try:
        for _ in range(2):
            check(lib().moea_algorithm_run(handle, ctypes.byref(ms)))
            view = _lib.PopulationViewC()
            check(lib().moea_algorithm_view(handle, ctypes.byref(view)))
            torch.cuda.synchronize()
            for p, shape in ((view.d_variables, (view.size, view.dimension)),
                             (view.d_objectives, (view.objectives, view.size))):
                from cuda_moea.algorithm import _view
                out.append(_view(p, shape, torch.float32, view.device, keep).clone())
            check(lib().moea_algorithm_reset(handle))
    finally:
        lib().moea_algorithm_destroy(handle)
    return out


@pytest.mark.parametrize("cls", [cm.NSGA3, cm.RVEA])
@pytest.mark.parametrize("N", [64, 1200])
def test_callback_problem_on_the_legacy_stream(cls, N):
    for a, b in zip(_run(cls, N, LEGACY_STREAM), _run(cls, N, None)):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
