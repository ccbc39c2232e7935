"""GPU: rows the BF16 bounds leave undecided, resolved 128 of a b view at a time.

Views made of dense clusters (copies of a few rows, apart by less than the bound)
leave every row undecided, with as many columns in its window as a cluster has:
counts of rows around a group's 128, columns around a tile's, shortlists below,
at and above their capacity, in single pairs (fewer groups than SMs) and in
batches (rows of many pairs in a group). Each list is the oracle's.
"""
import numpy as np
import pytest

import oracle as O
from skylens_match import synth

pytestmark = pytest.mark.gpu


def clustered(rng, n, per, sigma=0.004):
    base = synth.sift_like(rng, max(1, -(-n // per)))
    return synth.noisy_copy(rng, base[rng.permutation(np.arange(n) % len(base))], sigma)


def check(matcher, views, pairs, ratio, mutual, **kw):
    st = matcher.store(sum(len(v) for v in views), len(views))
    for v in views:
        st.add_view(v)
    plan = st.plan(pairs, ratio, mutual, "bf16", **kw)
    plan.launch()
    got = plan.per_pair()
    for k, (a, b) in enumerate(pairs):
        assert np.array_equal(got[k], O.ratio_match_np(views[a], views[b], ratio, mutual, threads=16)), (len(views[a]), len(views[b]))
    stats = plan.stats
    plan.close()
    st.close()
    return stats


@pytest.mark.parametrize("na,nb", [(1, 2), (16, 17), (127, 129), (128, 15), (129, 16), (257, 128), (300, 1300), (1300, 257), (2500, 3000)])
@pytest.mark.parametrize("mutual", [True, False])
def test_every_row_undecided(matcher, na, nb, mutual):
    rng = np.random.default_rng(na * 5000 + nb)
    b = clustered(rng, nb, 4)
    a = synth.noisy_copy(rng, b[rng.integers(0, nb, na)], 0.004)
    s = check(matcher, [a, b], [(0, 1)], 0.97, mutual)
    assert s["rows_rescored"] >= 0.8 * na and s["pairs_routed"] == 0


@pytest.mark.parametrize("per,routed", [(8, False), (24, False), (100, False), (127, False), (140, True), (400, True)])
def test_shortlists_around_their_capacity(matcher, per, routed):
    rng = np.random.default_rng(per)
    b = clustered(rng, 4 * per, per, 0.002)
    a = synth.noisy_copy(rng, b[rng.integers(0, len(b), 333)], 0.002)
    s = check(matcher, [a, b], [(0, 1)], 0.97, True)
    assert (s["pairs_routed"] == 1) == routed
    # a few rows above the capacity: scanned one by one
    c = np.concatenate([synth.sift_like(rng, 900), b])
    d = np.concatenate([synth.noisy_copy(rng, c[:880], 0.01), a[:60]])
    s = check(matcher, [d, c], [(0, 1), (1, 0)], 0.97, False)
    if routed:
        assert s["rows_recomputed"] >= 40


@pytest.mark.parametrize("n_views", [3, 12, 40])
def test_groups_of_many_pairs(matcher, n_views):
    rng = np.random.default_rng(n_views)
    base = clustered(rng, 260, 3)
    views = [synth.noisy_copy(rng, base[rng.integers(0, 260, int(rng.integers(1, 420)))], 0.004) for _ in range(n_views)]
    views[1] = views[1][:0].reshape(0, 128)
    pairs = [(a, b) for a in range(n_views) for b in range(max(0, a - 9), min(n_views, a + 9)) if a != b]
    s = check(matcher, views, pairs, 0.97, True)
    assert s["rows_rescored"] > 0


@pytest.mark.parametrize("k", [1, 8, 32])
def test_shortlist_capacity_asked_for(matcher, k):
    rng = np.random.default_rng(k)
    b = clustered(rng, 600, 20, 0.002)
    a = np.concatenate([synth.noisy_copy(rng, b[:30], 0.002), synth.noisy_copy(rng, synth.sift_like(rng, 500), 0.0)])
    s = check(matcher, [a, b], [(0, 1)], 0.97, True, shortlist_k=k)
    assert (s["rows_recomputed"] > 0) == (4 * k < 20)
