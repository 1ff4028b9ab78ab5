"""Hierarchical clustering on the device (spops_pairs_cluster): the same
permutation and offsets as the host loop (csrc/hc.cpp) and the reference's
hierarchical_clustering_v0_fast (include/spgemm_utility.h:742-915), bit for
bit, on LSH pairs of planted-community matrices, on rows in groups that
produce long merge chains and pairs found while merging, and on random pair
lists whose scores tie often."""
import numpy as np
import pytest

from sparseops_b200 import synth

pytestmark = pytest.mark.gpu


def _csr(rp, ci, ncols):
    import torch
    from sparseops_b200 import CSR_Matrix
    d = torch.device("cuda")
    return CSR_Matrix(len(rp) - 1, ncols, torch.from_numpy(rp).to(d), torch.from_numpy(ci).to(d),
                      torch.ones(len(ci), dtype=torch.float64, device=d))


def _check(rp, ci, ncols, cluster_size, ref):
    from sparseops_b200.spgemm import (hierarchical_clustering_device, hierarchical_clustering_v0_fast,
                                       lsh_candidate_pairs_vector)
    A = _csr(rp, ci, ncols)
    pairs = lsh_candidate_pairs_vector(A, 64, 16, 7)
    n = len(rp) - 1
    hperm, hoffs = hierarchical_clustering_v0_fast(rp, ci, n, pairs, cluster_size)
    dperm, doffs = hierarchical_clustering_device(A, pairs, cluster_size)
    assert np.array_equal(dperm, hperm) and np.array_equal(doffs, hoffs)
    pi, pj, ps = pairs.host()
    rperm, roffs = ref.hc(rp, ci, pi, pj, ps, cluster_size)
    assert np.array_equal(dperm, rperm) and np.array_equal(doffs, roffs)
    return len(doffs) - 1


@pytest.mark.parametrize("n,ncomm,cs", [(16384, 64, 8), (131072, 512, 8), (131072, 512, 3)])
def test_device_hc_planted(cuda, ref, n, ncomm, cs):
    rp, ci, _ = synth.planted_communities(n, ncomm=ncomm, mean=20.0, seed=17)
    _check(rp, ci, n, cs, ref)


@pytest.mark.parametrize("group,width,cs", [(32, 12, 8), (64, 16, 8), (16, 8, 4), (128, 24, 14)])
def test_device_hc_grouped(cuda, ref, group, width, cs):
    """Near-duplicate rows in groups: many tasks competing for few clusters,
    and pairs found while merging."""
    n = 65536
    rp, ci, _, nc = synth.grouped_rows(n, group=group, width=width, seed=group + width)
    assert _check(rp, ci, nc, cs, ref) < n  # clusters did form


def test_device_hc_random_pairs(cuda, ref):
    """Random pair lists (sorted, i < j, unique) with scores from a handful of
    values, so equal scores break ties on (i, j)."""
    from sparseops_b200.spgemm import hierarchical_clustering_device, hierarchical_clustering_v0_fast, pairs_from_arrays
    rng = np.random.default_rng(5)
    for trial in range(6):
        n = int(rng.integers(50, 3000))
        rp, ci, _ = synth.planted_communities(n, ncomm=max(1, n // 40), mean=6.0, seed=100 + trial)
        m = int(rng.integers(10, 6 * n))
        a, b = rng.integers(0, n, m), rng.integers(0, n, m)
        keep = a != b
        a, b = np.minimum(a[keep], b[keep]), np.maximum(a[keep], b[keep])
        key = np.unique(a * n + b)
        pi, pj = key // n, key % n
        ps = rng.integers(0, 9, len(pi)) / 8.0
        cs = int(rng.integers(2, 10))
        hperm, hoffs = hierarchical_clustering_v0_fast(rp, ci, n, (pi, pj, ps), cs)
        rperm, roffs = ref.hc(rp, ci, pi, pj, ps, cs)
        assert np.array_equal(hperm, rperm) and np.array_equal(hoffs, roffs)
        dperm, doffs = hierarchical_clustering_device(_csr(rp, ci, n), pairs_from_arrays(pi, pj, ps), cs)
        assert np.array_equal(dperm, hperm) and np.array_equal(doffs, hoffs), trial


def test_device_hc_unsorted_pairs_take_the_host_loop(cuda):
    """A pair list that is not sorted i < j pairs gives the host loop's result."""
    from sparseops_b200.spgemm import hierarchical_clustering_device, hierarchical_clustering_v0_fast, pairs_from_arrays
    rp, ci, _ = synth.planted_communities(2000, ncomm=40, mean=6.0, seed=9)
    pi = np.array([5, 3, 7, 100], np.int64)
    pj = np.array([9, 1, 8, 50], np.int64)
    ps = np.array([0.5, 0.5, 0.25, 0.75])
    hperm, hoffs = hierarchical_clustering_v0_fast(rp, ci, 2000, (pi, pj, ps), 4)
    dperm, doffs = hierarchical_clustering_device(_csr(rp, ci, 2000), pairs_from_arrays(pi, pj, ps), 4)
    assert np.array_equal(dperm, hperm) and np.array_equal(doffs, hoffs)


@pytest.mark.parametrize("sizes", [
    [(2, 1), (3, 3), (32, 496), (33, 500), (64, 512), (64, 513), (65, 512)],       # one-warp blocks and just above
    [(256, 8192), (256, 8193), (257, 300), (255, 1000), (2, 1), (64, 63)],         # 256-thread blocks and just above
    [(1500, 4000), (700, 699), (64, 400), (20, 30), (2, 1)],                       # the rounds beside both
])
@pytest.mark.parametrize("cs", [2, 8, 40])
def test_device_hc_component_sizes(cuda, sizes, cs):
    """Connected components of given (rows, pairs) at the limits between the
    block forms and the rounds, over rows in random order, with tied scores."""
    from sparseops_b200.spgemm import hierarchical_clustering_device, hierarchical_clustering_v0_fast, pairs_from_arrays
    rng = np.random.default_rng(sum(r + p for r, p in sizes) + cs)
    n = sum(r for r, _ in sizes) + 37  # some rows in no pair
    rows = rng.permutation(n)
    key, at = [], 0
    for r, p in sizes:
        mine, at = rows[at:at + r], at + r
        have = {(min(a, b), max(a, b)) for a, b in zip(mine[:-1], mine[1:])}  # a path connects them
        while len(have) < p:
            a, b = rng.choice(mine, 2, replace=False)
            have.add((min(a, b), max(a, b)))
        key += [int(a) * n + int(b) for a, b in have]
    key = np.sort(np.array(key, np.int64))
    pi, pj = key // n, key % n
    ps = rng.integers(0, 17, len(key)) / 16.0
    rp, ci, _ = synth.planted_communities(n, ncomm=max(1, n // 40), mean=6.0, seed=n)
    hperm, hoffs = hierarchical_clustering_v0_fast(rp, ci, n, (pi, pj, ps), cs)
    dperm, doffs = hierarchical_clustering_device(_csr(rp, ci, n), pairs_from_arrays(pi, pj, ps), cs)
    assert np.array_equal(dperm, hperm) and np.array_equal(doffs, hoffs)


@pytest.mark.parametrize("sizes", [
    [(32, 256), (32, 257), (33, 256), (33, 40), (2, 1)],              # both sides of the four-warp blocks' limits
    [(31, 200), (32, 31), (16, 120), (23, 253), (2, 1), (5, 4)] * 2,  # those blocks alone, not all warps in use
    [(9, 20)] * 9 + [(64, 512), (256, 4000), (2, 1)],                 # all three forms at once
])
@pytest.mark.parametrize("cs", [2, 8, 40])
def test_device_hc_tiny_component_sizes(cuda, sizes, cs):
    """As test_device_hc_component_sizes, at the limits of the four-warp form."""
    test_device_hc_component_sizes(cuda, sizes, cs)
