"""The sampler's candidate path for the top-k pivot (ops/csrc/sampling.cu), restated with numpy:
the k-th largest of the 256 group maxima is a lower bound of the k-th largest value, so the
entries at or above it contain the whole top-k set and the pivot can be picked among them."""
import numpy as np
import pytest

THREADS, GROUPS = 1024, 256


def _pivot_by_candidates(row: np.ndarray, k: int, aligned: bool = True):
    v = len(row)
    # group g takes the 16-byte pieces g, g + 256, ..., or the elements where a group would get no piece;
    # a large vocabulary goes round the threads, of which four lanes 8 apart make a group, and so does
    # the ragged end
    gmax = np.full(GROUPS, -np.inf)
    spread = v < 16 * THREADS
    piece = 4 if aligned and (not spread or v >= 4 * GROUPS) else 1
    body = v // piece * piece
    top = row[:body].reshape(-1, piece).max(axis=1)
    t = np.arange(len(top)) % THREADS
    at = np.arange(len(top)) % GROUPS if spread else (t >> 5) * 8 + (t & 7)
    np.maximum.at(gmax, at, top)
    t = np.arange(v - body)
    np.maximum.at(gmax, (t >> 5) * 8 + (t & 7), row[body:])
    # rank by (value desc, group index asc): the group of rank k - 1 gives the bound
    order = sorted(range(GROUPS), key=lambda j: (-gmax[j], j))
    bound = gmax[order[k - 1]]
    cand = row[row >= bound]
    # the candidate with fewer than k values above it and at least k at or above it
    pivots = {c for c in cand if (cand > c).sum() < k <= (cand >= c).sum()}
    assert len(pivots) == 1
    return pivots.pop(), len(cand), v


@pytest.mark.parametrize("seed", range(12))
@pytest.mark.parametrize("k", [1, 5, 50, 256])
def test_candidate_pivot_is_the_kth_largest(seed, k):
    rng = np.random.default_rng(seed)
    v = int(rng.choice([1500, 32016, 40000]))
    row = rng.standard_normal(v).astype(np.float32) * 2
    if seed % 3 == 0:                       # ties, also at the pivot
        row[rng.integers(0, v, 200)] = 3.25
        row[rng.integers(0, v, 40)] = 9.0
    pivot, n_cand, _ = _pivot_by_candidates(row, k)
    assert pivot == np.sort(row)[-k]
    assert n_cand >= k
    if seed % 3 and k < 256:
        assert n_cand <= (512 if v < 16 * THREADS else 1024)    # short enough to be ranked


@pytest.mark.parametrize("v", [500, 1000, 1024, 2000, 4000, 4096, 5003])
@pytest.mark.parametrize("aligned", [True, False])
def test_small_vocabularies_leave_few_candidates(v, aligned):
    """No group is empty where there are 256 elements: with as many groups as top_k or more the bound
    still drops most of the row."""
    for seed in range(6):
        row = np.random.default_rng(seed).standard_normal(v).astype(np.float32)
        for k, share in ((50, 0.25), (200, 0.8)):
            pivot, n_cand, _ = _pivot_by_candidates(row, k, aligned)
            assert pivot == np.sort(row)[-k]
            assert n_cand <= share * v
