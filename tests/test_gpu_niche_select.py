"""GPU: the generation's niche selection (direction buckets in one cluster,
the sorts for buckets too large to be ranked by counting) against the oracle's
three stable sorts: survivors, sizes and the random-word counter are equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _selection(n, H, seed, spread):
    rng = np.random.default_rng(seed)
    if spread:   # mutually non-dominated: the last front is the population
        f = rng.random((3, n)) + 1e-3
        objs = f / np.linalg.norm(f, axis=0)
    else:        # several fronts, integer-valued objectives (ties, equal distances)
        objs = rng.integers(1, 12, (3, n)).astype(np.float64)
    d = rng.random((3, H)) + 1e-3
    return objs.astype(np.float32), (d / np.linalg.norm(d, axis=0)).astype(np.float32)


# One to sixteen CTAs at their boundaries; one direction with more members than
# a bucket may hold (sorts), with as many (levels beyond the histogram) and
# with few; more directions than points.
@pytest.mark.parametrize("n,H,spread", [
    (2, 1, True), (62, 91, True), (1024, 40, True), (1026, 1, True), (2048, 1, True), (2050, 2, True),
    (4096, 3, True), (4098, 1, True), (4098, 5000, True), (9000, 2, True), (20000, 6, False), (300, 9000, False),
    (65536, 900, True)])
def test_niche_selection_matches_oracle(n, H, spread):
    from cuda_moea import stages as st
    from oracle import oracle as O
    objs, refs = _selection(n, H, n + H, spread)
    cv = np.zeros(n, np.float32)
    ideal = objs[:, : n // 2].min(1)
    ws = st.Workspace(n, 3, H)
    want = O.nsga3_select(cv, objs, refs, 77, 5, ideal)
    for _ in range(2):  # the second call finds the first one's scratch
        got = st.nsga3_select(ws, torch.from_numpy(cv).cuda(), torch.from_numpy(objs).cuda(),
                              torch.from_numpy(refs).cuda(), 77, 5, torch.from_numpy(ideal).cuda(), st.ASSOC_SCAN)
        np.testing.assert_array_equal(got["sizes"].cpu().numpy(), want["sizes"])
        np.testing.assert_array_equal(got["survivors"].cpu().numpy(), want["survivors"])
        assert got["offset"] == want["offset"]
