"""GPU: the exact FP32 kernel at the edges of its row and column groups of 32.

Sizes around every multiple of 32 up to one past two tiles, all against all, in
one batch (many pairs and views without rows between them share the persistent
CTAs), with exact ties inside and across tiles, rows that are infinite or NaN,
and the cross-check on and off. Every list must equal the oracle's.
"""
import numpy as np
import pytest

import oracle as O
from skylens_match import synth

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 255, 257]


@pytest.fixture(scope="module")
def views():
    rng = np.random.Generator(np.random.PCG64(97))
    base = synth.sift_like(rng, 300)
    out = []
    for n in SIZES:
        k = n // 2
        v = np.concatenate([synth.noisy_copy(rng, base[rng.permutation(300)[:k]], 0.05), synth.sift_like(rng, n - k)])
        v = v[rng.permutation(n)] if n else v.reshape(0, 128)
        if n > 40:  # equal rows: the lowest index wins, within and across tiles
            v[n - 1] = v[0]
            v[33] = v[7]
        out.append(np.ascontiguousarray(v, dtype=np.float32))
    return out


@pytest.mark.parametrize("mutual", [True, False])
def test_all_sizes_in_one_batch(matcher, views, mutual):
    st = matcher.store(sum(len(v) for v in views), len(views))
    ids = [st.add_view(v) for v in views]
    pairs = [(a, b) for a in ids for b in ids if a != b]
    plan = st.plan(pairs, 0.8, mutual, "fp32")
    plan.launch()
    got = plan.per_pair()
    for k, (a, b) in enumerate(pairs):
        want = O.ratio_match_np(views[a], views[b], 0.8, mutual, threads=16)
        assert np.array_equal(got[k], want), (SIZES[a], SIZES[b], mutual)
    plan.close()
    st.close()


@pytest.mark.parametrize("n", [33, 97, 130, 257])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("mutual", [True, False])
def test_rows_that_are_not_finite(matcher, views, n, bad, mutual):
    rng = np.random.Generator(np.random.PCG64(n))
    b = synth.sift_like(rng, n)
    a = synth.noisy_copy(rng, b[rng.permutation(n)], 0.05)
    for v, rows in ((a, (0, n - 1)), (b, (5, n // 2, n - 2))):
        for r in rows:
            v[r, rng.integers(0, 128)] = bad
    want = O.ratio_match_np(a, b, 0.8, mutual, threads=16)
    assert np.array_equal(matcher.ratio_match_np(a, b, 0.8, mutual, "fp32"), want)


@pytest.mark.parametrize("na,nb", [(31, 33), (64, 96), (129, 255), (257, 700), (700, 257), (1, 1500), (1500, 2),
                                   (1000, 1000), (1700, 1300)])
def test_items_of_part_of_a_tile(matcher, na, nb):
    # few tiles: items of one 32 x 32 block up to a tile, by the call's size; the
    # pair alone and with others in a plan
    rng = np.random.Generator(np.random.PCG64(na * 4099 + nb))
    b = synth.sift_like(rng, nb)
    k = min(na, nb) // 2
    a = np.concatenate([synth.noisy_copy(rng, b[rng.permutation(nb)[:k]], 0.05), synth.sift_like(rng, na - k)])
    want = {m: O.ratio_match_np(a, b, 0.8, m, threads=16) for m in (True, False)}
    for mutual in (True, False):
        assert np.array_equal(matcher.ratio_match_np(a, b, 0.8, mutual, "fp32"), want[mutual])
    st = matcher.store(na + nb + 200, 3)
    ids = [st.add_view(v) for v in (a, b, synth.sift_like(rng, 70))]
    plan = st.plan([(ids[0], ids[1]), (ids[2], ids[0]), (ids[0], ids[1])], 0.8, True, "fp32")
    plan.launch()
    got = plan.per_pair()
    assert np.array_equal(got[0], want[True]) and np.array_equal(got[2], want[True])
    plan.close()
    st.close()
