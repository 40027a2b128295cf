"""GPU: batches whose groups (and batches side by side whose instances) need
different amounts of shared memory for the offspring rows, both above the
default limit of a launch: every instance equals the one run alone."""
import threading

import pytest
import torch

import cuda_moea as cm

pytestmark = pytest.mark.gpu


def _make(N, D, kind="DTLZ2", T=4):
    return cm.NSGA3(population_size=N, max_generations=T, problem=getattr(cm, kind)(D, 3), seed=N + D,
                    print_progress=False)


def _equals_alone(batch, i, N, D, kind="DTLZ2"):
    want, got = _make(N, D, kind).run(), batch.result(i)
    assert torch.equal(got.variables.view(torch.int32), want.variables.view(torch.int32))
    assert torch.equal(got.objectives.contiguous().view(torch.int32), want.objectives.contiguous().view(torch.int32))


# D = 258: 256 g-terms, the most of the fused generation; D = 193: the first above 48 KB
@pytest.mark.parametrize("dims", [(258, 200), (200, 258), (258, 193), (193, 258), (258, 12), (12, 258)])
def test_groups_of_different_row_lengths(dims):
    sizes = (200, 100)  # the larger population takes the first group
    batch = cm.Batch([_make(N, D) for N, D in zip(sizes, dims)], groups=2)
    assert batch.fused and batch.schedule["groups"] == 2
    batch.run()
    for i, (N, D) in enumerate(zip(sizes, dims)):
        _equals_alone(batch, i, N, D)


@pytest.mark.parametrize("dims", [(258, 200), (200, 258)])
def test_batches_of_different_row_lengths_side_by_side(dims):
    batches = [cm.Batch([_make(100, D), _make(60, D)]) for D in dims]
    for _ in range(4):
        for b in batches:
            b.step()
    for b, D in zip(batches, dims):
        b.synchronize()
        _equals_alone(b, 0, 100, D)
        _equals_alone(b, 1, 60, D)


def test_batches_of_different_row_lengths_from_two_threads():
    """Each thread captures and runs batches of its own row length."""
    errors = []

    def work(D):
        try:
            for _ in range(150):
                b = cm.Batch([_make(8, D)])
                b.run(2)
                b.close()
        except Exception as e:  # noqa: BLE001 - reported by the test
            errors.append((D, e))
    threads = [threading.Thread(target=work, args=(D,)) for D in (258, 193)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
