"""The one-launch search of a few queries (scan, per-CTA lists, merge by the last CTA): parity with the oracle at the edges
of its rounds, lists and merge."""
import numpy as np
import pytest

import oracle
from parity import assert_topk_parity

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vsk():
    import vectorstorekit_b200 as v
    return v


@pytest.fixture(scope="module")
def dev(vsk):
    return vsk.CUDAAcceleratorStrategy(0).initialize()


METRICS = {"euclidean": oracle.EUCLIDEAN, "cosine": oracle.COSINE, "dotProduct": oracle.DOT, "manhattan": oracle.MANHATTAN}


def _index(vsk, dev, metric, x, masks=None):
    ix = vsk.FlatIndex(dev, x.shape[1], vsk.DistanceMetric(metric))
    ix.add(x, masks)
    return ix


# fewer rows than k, one warp step, one CTA, partial rounds, several rounds per CTA; 1, 2, 4 and 8 staged queries;
# widths with 16-byte loads and without, around one and two steps of a warp; k up to the path's limit
@pytest.mark.parametrize("metric", list(METRICS))
@pytest.mark.parametrize("shape", [(1, 8, 1, 3), (15, 128, 1, 10), (33, 5, 2, 33), (1_000, 131, 3, 128), (10_000, 128, 1, 10),
                                   (70_001, 96, 1, 100), (200_000, 33, 8, 128), (30_001, 260, 5, 1), (9_999, 1_536, 8, 7)])
def test_few_queries(vsk, dev, cpu_oracle, metric, shape):
    n, d, nq, k = shape
    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d)).astype(np.float32)
    q = rng.standard_normal((nq, d)).astype(np.float32)
    ix = _index(vsk, dev, metric, x)
    ix2 = _index(vsk, dev, metric, x, np.full(n, 3, np.uint64))
    rd, ri = cpu_oracle.flat_search(METRICS[metric], q, x, min(k, n))
    for got in (ix.batchSearch(q, min(k, n)), ix2.batchSearch(q, min(k, n), np.full(nq, 2, np.uint64))):
        assert_topk_parity(got[0], got[1], rd, ri)
    if k > n:
        d_, i_ = ix.batchSearch(q, k)
        assert np.all(i_[:, n:] == -1) and np.all(np.isinf(d_[:, n:]))


# one query: widths around the short-row forms and around what travels in the launch's arguments; lists handed over whole (96 keys)
# and shortened; the query on the host and on the device
@pytest.mark.parametrize("metric", list(METRICS))
@pytest.mark.parametrize("shape", [(20_003, 128, 96), (20_003, 132, 97), (40_001, 256, 10), (9_001, 260, 128), (3_001, 1_024, 5), (3_001, 1_028, 128),
                                   (120_001, 4, 128)])
def test_one_query(vsk, dev, cpu_oracle, metric, shape):
    import torch
    n, d, k = shape
    rng = np.random.default_rng(n + d + k)
    x = rng.standard_normal((n, d)).astype(np.float32)
    q = rng.standard_normal((1, d)).astype(np.float32)
    ix = _index(vsk, dev, metric, x)
    got = ix.batchSearch(q, k)
    assert_topk_parity(*got, *cpu_oracle.flat_search(METRICS[metric], q, x, k))
    on_device = ix.batchSearch(torch.from_numpy(q).cuda(), k)
    assert np.array_equal(got[0], on_device[0].cpu().numpy()) and np.array_equal(got[1], on_device[1].cpu().numpy())


def test_merge_of_lists_within_the_bound(vsk, dev, cpu_oracle):
    """Rows that all tie at one distance but for a few: every key of every list is within the merge's bound."""
    x = np.zeros((60_000, 64), np.float32)
    x[::1_000, 0] = 1.0
    ix = _index(vsk, dev, "euclidean", x)
    q = np.zeros((1, 64), np.float32)
    for k in (1, 50, 128):
        d_, i_ = ix.batchSearch(q, k)
        rd, ri = cpu_oracle.flat_search(oracle.EUCLIDEAN, q, x, k)
        assert np.array_equal(i_, ri) and np.array_equal(d_, rd)


@pytest.mark.parametrize("order", ["ascending", "descending", "blocks"])
def test_order_of_rows_and_ties(vsk, dev, cpu_oracle, order):
    """Rows sorted by distance (every later row is listed, or none is), the nearest rows all in one CTA's share, and bulk
    ties: the result is the first k by (distance, id)."""
    n, d, k = 60_000, 16, 128
    t = np.repeat(np.arange(n // 50, dtype=np.float32), 50)      # 50 rows tie at every distance
    if order == "descending":
        t = t[::-1].copy()
    if order == "blocks":
        t = np.roll(t, 1_234)
    x = np.zeros((n, d), np.float32)
    x[:, 3] = t
    ix = _index(vsk, dev, "euclidean", x)
    q = np.zeros((2, d), np.float32)
    q[1, 3] = 700.0
    for m in (1, 2):
        d_, i_ = ix.batchSearch(q[:m], k)
        rd, ri = cpu_oracle.flat_search(oracle.EUCLIDEAN, q[:m], x, k)
        assert np.array_equal(i_, ri) and np.array_equal(d_, rd)


def test_filters_few_rows_pass(vsk, dev, cpu_oracle):
    rng = np.random.default_rng(4)
    n, d = 40_000, 64
    x = rng.standard_normal((n, d)).astype(np.float32)
    masks = np.zeros(n, np.uint64)
    masks[rng.choice(n, 25, replace=False)] = 1
    masks[7::1000] |= np.uint64(2)
    q = rng.standard_normal((4, d)).astype(np.float32)
    qm = np.array([1, 2, 4, 3], np.uint64)
    d_, i_ = _index(vsk, dev, "manhattan", x, masks).batchSearch(q, 50, qm)
    for r in range(4):
        rows = np.nonzero(masks & qm[r])[0]
        assert np.all(i_[r, len(rows):] == -1)
        if len(rows):
            m = min(50, len(rows))
            rd, ri = cpu_oracle.flat_search(oracle.MANHATTAN, q[r:r + 1], x[rows], m)
            assert_topk_parity(d_[r:r + 1, :m], i_[r:r + 1, :m], rd, rows[ri])


def test_repeated_calls_leave_the_tickets_at_zero(vsk, dev, cpu_oracle):
    """Back-to-back calls of different grids on one context, a probe of inverted lists among them."""
    rng = np.random.default_rng(5)
    x = rng.standard_normal((20_000, 32)).astype(np.float32)
    big, small = _index(vsk, dev, "euclidean", x), _index(vsk, dev, "dotProduct", x[:100])
    ivf = vsk.IVFIndex(dev, 32, 64, 64, maxIterations=2)
    ivf.train(x[:4_096], x[:64])
    ivf.insert(x)
    for r in range(6):
        q = rng.standard_normal((1 + 2 * (r % 2), 32)).astype(np.float32)
        rd, ri = cpu_oracle.flat_search(oracle.EUCLIDEAN, q, x, 20)
        assert_topk_parity(*big.batchSearch(q, 20), rd, ri)
        assert_topk_parity(*ivf.batchSearch(q, 20), rd, ri)      # every list is probed: the flat result
        rd, ri = cpu_oracle.flat_search(oracle.DOT, q, x[:100], 5)
        assert_topk_parity(*small.batchSearch(q, 5), rd, ri)


@pytest.fixture(scope="module")
def large():
    """Rows beyond the line from which the fp16 copy is read; row 7 twice, and a nearest row 1 500 times for one query."""
    rng = np.random.default_rng(6)
    x = rng.standard_normal((110_000, 1_300), dtype=np.float32)
    x[90_000] = x[7]
    q = rng.standard_normal((6, 1_300), dtype=np.float32)
    q[1] = x[7] + 0.01
    q[4] = x[500] * 1.1
    x[60_000:61_500] = x[500]
    return x, q


@pytest.mark.parametrize("metric", ["euclidean", "cosine", "dotProduct"])
@pytest.mark.parametrize("nq,k", [(1, 10), (3, 100), (6, 128)])
def test_large_store_reads_the_fp16_copy(vsk, dev, cpu_oracle, large, metric, nq, k):
    x, q = large
    ix = _index(vsk, dev, metric, x)
    before = dev.stats()
    got = ix.batchSearch(q[:nq], k)
    after = dev.stats()
    assert after["tensor_tiles"] == before["tensor_tiles"]
    assert (after["fallback_queries"] > before["fallback_queries"]) == (nq > 4)    # 1 500 equal rows fill one query's list
    assert_topk_parity(*got, *cpu_oracle.flat_search(METRICS[metric], q[:nq], x, k))
    ix.close()


# batches on the list tiles of which a few queries overflow: the last step walks the lists of those alone, by number
@pytest.mark.parametrize("d,nbad", [(16, 1), (16, 17), (40, 3), (40, 64), (40, 65)])
def test_overflowed_queries_of_an_inverted_file_batch(vsk, dev, cpu_oracle, d, nbad):
    rng = np.random.default_rng(d + nbad)
    n, nlist, nq, k = 120_000, 8, 300, 10
    centres = 4.0 * rng.standard_normal((nlist, d)).astype(np.float32)
    x = (centres[rng.integers(0, nlist, n)] + rng.standard_normal((n, d))).astype(np.float32)
    x[60_000:66_000] = centres[0] + 0.3                           # 6 000 equal rows
    q = (centres[rng.integers(1, nlist, nq)] + rng.standard_normal((nq, d))).astype(np.float32)
    hit = rng.choice(nq, nbad, replace=False)
    q[hit] = centres[0] + 0.3 + 1e-3 * rng.standard_normal((nbad, d)).astype(np.float32)
    ivf = vsk.IVFIndex(dev, d, nlist, 2, maxIterations=4, tolerance=-1.0)
    ivf.train(x[:20_000], centres.copy())
    ivf.insert(x)
    before = dev.stats()
    got = ivf.batchSearch(q, k)
    after = dev.stats()
    assert after["tensor_tiles"] > before["tensor_tiles"]
    # (the list tiles, which take more than 64 of them, overflow once more and count it)
    again = after["fallback_queries"] - before["fallback_queries"]
    assert again == nbad if nbad <= 64 else again >= nbad
    assert_topk_parity(*got, *cpu_oracle.ivf_search(q, x, ivf.centroids, ivf.assignments(), 2, k))
    ivf.close()


def test_probes_of_short_rows_take_one_launch(vsk, dev, cpu_oracle):
    """Up to sixteen queries over rows of at most 32 dimensions: the probe selection, and the walk of re-run queries, have no
    reason to keep to the chunked schedule (the lists themselves do, and count what overflows there)."""
    rng = np.random.default_rng(9)
    x = rng.standard_normal((30_000, 24)).astype(np.float32)
    ivf = vsk.IVFIndex(dev, 24, 64, 64, maxIterations=2)
    ivf.train(x[:4_096], x[:64])
    ivf.insert(x)
    for nq in (3, 8, 16):
        q = rng.standard_normal((nq, 24)).astype(np.float32)
        assert_topk_parity(*ivf.batchSearch(q, 20), *cpu_oracle.flat_search(oracle.EUCLIDEAN, q, x, 20))


# 1, 2, 8 and 16 queries walk both lists in several rounds per CTA (the launch's CTAs, three per SM, are shared by the queries, and
# a round is 512 rows of a CTA): on 148 SMs the nearer list takes 3.5 rounds, 4, 5 and 5.
@pytest.mark.parametrize("nq,d,n,launches", [(1, 8, 1_200_000, 2), (2, 8, 700_000, 3), (8, 36, 210_000, 3), (16, 36, 105_000, 5)])
def test_listed_rows_get_their_ids_in_every_round(vsk, dev, nq, d, n, launches):
    """Every row of the nearer list is nearer than all before it, so that each is listed, most of them in the rounds after the
    first; every third row belongs to the other list, so that no stored row's number is its id.  Against the order of insertion."""
    import torch
    k = 100
    far = np.arange(n) % 3 == 0
    x = np.zeros((n, d), np.float32)
    x[~far, 1] = np.arange((~far).sum(), 0, -1)                  # whole numbers; the last rows are the nearest
    x[far, 1] = 2e7
    cent = np.zeros((2, d), np.float32)
    cent[1, 1] = 2e7
    q = np.zeros((nq, d), np.float32)
    q[:, 2] = np.arange(nq)                                      # (off the rows' line: the same order for every query)
    ix = vsk.IVFIndex(dev, d, numberOfCentroids=2, numberOfProbes=2)
    ix.centroids, ix.trained = cent, True
    ix.insert(x)
    ids = np.nonzero(~far)[0][:-k - 1:-1]
    dist = np.sqrt(np.arange(1, k + 1) ** 2 + np.arange(nq)[:, None] ** 2).astype(np.float32)   # (sums below 2^24)
    for _ in range(20):
        before = dev.stats()["kernel_launches"]
        gd, gi = (a.cpu().numpy() for a in ix.batchSearch(torch.from_numpy(q).cuda(), k))
        assert dev.stats()["kernel_launches"] - before == launches   # the probe list (merged apart from two queries on), and the walk
        assert np.array_equal(gi, np.tile(ids, (nq, 1))) and np.allclose(gd, dist, rtol=2e-7, atol=0)
    ix.close()
