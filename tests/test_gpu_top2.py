"""GPU: the BF16 pass's per-row (nearest, second nearest) at the edges of its
tiles, steps, chunks and classes.

A row keeps the minima of 16-column chunks and of the 16 column classes; the
second nearest column may share the nearest one's chunk, its class, or
neither. Columns end anywhere within a 16-column chunk, a 128-row tile and a
two-tile step. Each list must equal the oracle's.
"""
import numpy as np
import pytest

import oracle as O
from skylens_match import synth

pytestmark = pytest.mark.gpu


def pair(seed, na, nb):
    """b: noisy copies of rows of a, each with a rival at distance 1 (the same
    chunk, most often), 16 (the same class), 5 or 128 columns further: exact
    and near duplicates of the copy, so that second best and ties fall there."""
    rng = np.random.Generator(np.random.PCG64(seed))
    a, b = synth.sift_like(rng, na), synth.sift_like(rng, nb)
    for n, j in enumerate(range(0, nb, 7)):
        b[j] = synth.noisy_copy(rng, a[rng.integers(na)][None], 0.04)[0]
        rival = j + (1, 16, 5, 128)[n % 4]
        if rival < nb and n % 3:
            b[rival] = b[j] if n % 2 else synth.noisy_copy(rng, b[j][None], (0.002, 0.03)[n % 5 > 2])[0]
    return a, b


@pytest.mark.parametrize("mutual", [True, False])
@pytest.mark.parametrize("na,nb", [(1, 2), (2, 1), (1, 16), (1, 17), (129, 15), (130, 31), (255, 33), (256, 128), (257, 257),
                                   (300, 272), (513, 511), (128, 1040), (1500, 260)])
def test_edges_equal_the_oracle(matcher, na, nb, mutual):
    for ratio in (0.8, 0.99):
        a, b = pair(na * 1000 + nb, na, nb)
        got = matcher.ratio_match_np(a, b, ratio, mutual, "bf16")
        assert np.array_equal(got, O.ratio_match_np(a, b, ratio, mutual, threads=8)), ratio


@pytest.mark.parametrize("n", [20, 700, 3000])
def test_undecided_rows_of_shared_and_large_views(matcher, n):
    """Rows whose ratio test hangs on less than the bound, from several a views
    against one b view (one undecided list), with few and many columns (one CTA
    a group, a cluster of them), and more of them than one group holds."""
    rng = np.random.Generator(np.random.PCG64(n))
    b = synth.sift_like(rng, n)
    d2 = ((b[:200, None] - b[None]) ** 2).sum(-1)
    d2[np.arange(len(d2)), np.arange(len(d2))] = 9.0
    views = [b]
    for v in range(3):
        # rows on the segment to their nearest neighbour, where d1 = 0.64 d2 up to the noise
        k = rng.integers(0, len(d2), 90)
        t = (0.8 / 1.8 + rng.normal(0, 0.004, 90)).astype(np.float32)[:, None]
        views.append(np.ascontiguousarray(b[k] * (1 - t) + b[d2[k].argmin(1)] * t, dtype=np.float32))
    st = matcher.store(sum(len(v) for v in views), len(views))
    for v in views:
        st.add_view(v)
    pairs = [(1, 0), (2, 0), (3, 0), (0, 1), (1, 0)]
    plan = st.plan(pairs, 0.8, True, "bf16")
    for _ in range(2):
        plan.launch()
        for (u, v), got in zip(pairs, plan.per_pair()):
            assert np.array_equal(got, O.ratio_match_np(views[u], views[v], 0.8, True, threads=8)), (u, v)
    assert plan.stats["rows_rescored"] + plan.stats["rows_recomputed"] > 50
    plan.close()
    st.close()


@pytest.mark.parametrize("na,nb", [(300, 112000), (100, 336000), (5800, 5800)])
@pytest.mark.parametrize("kind", ["sift", "sparse"])
def test_fp8_pairs_above_the_sample_threshold(matcher, kind, na, nb):
    """Pairs just above 2^25 distances: their sample decides whether FP8 pass 1
    runs. SIFT-like ones are rescued by it; sparse ones (one to three large
    components, distances far apart) need not be. Either way the oracle's list."""
    rng = np.random.Generator(np.random.PCG64(na))
    if kind == "sift":
        a, b = synth.sift_like(rng, na), synth.sift_like(rng, nb)
    else:
        def sparse(n):
            x = np.zeros((n, 128), np.float32)
            for _ in range(3):
                x[np.arange(n), rng.integers(0, 128, n)] = rng.integers(1, 9, n)
            return x
        a, b = sparse(na), sparse(nb)
    k = min(na, 64)
    b[rng.permutation(nb)[:k]] = a[:k] + np.float32(0.01) * rng.standard_normal((k, 128), dtype=np.float32)
    got = matcher.ratio_match_np(a, b, 0.8, True, "fp8")
    assert np.array_equal(got, O.ratio_match_np(a, b, 0.8, True, threads=16))
    if kind == "sift":
        assert matcher.last_stats["pairs_rescued"] == 1
