"""Manhattan batches through the byte filter (vabsdiff4 sums bound the fp32 distances, listed rows are re-scored): the rows
the CPU oracle finds, for partial tiles, widths around the 16-byte pieces and 64-byte chunks, filters and hostile data."""
import numpy as np
import pytest

import oracle
from parity import assert_topk_parity, logged_launches

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vsk():
    import vectorstorekit_b200 as v
    return v


@pytest.fixture(scope="module")
def dev(vsk):
    return vsk.CUDAAcceleratorStrategy(0).initialize()


def _index(vsk, dev, x, masks=None):
    ix = vsk.FlatIndex(dev, x.shape[1], vsk.DistanceMetric.manhattan)
    ix.add(x, masks)
    return ix


# every query tile (32, 64, 128), the smallest batch and index, partial query and row tiles, one and several chunks of
# bytes, widths that are not multiples of 4 or 16, k up to the path's limit
@pytest.mark.parametrize("shape", [(16_384, 256, 32, 50), (16_385, 64, 33, 1), (20_001, 65, 64, 10), (17_001, 5, 130, 10),
                                   (30_000, 100, 128, 100), (18_000, 512, 250, 37), (40_000, 16, 96, 1024), (50_001, 250, 40, 10)])
def test_byte_filter_finds_the_oracles_rows(vsk, dev, cpu_oracle, shape):
    n, d, nq, k = shape
    rng = np.random.default_rng(n + d)
    x = (rng.uniform(-1, 1, (n, d)) + rng.normal(0, 3, d)).astype(np.float32)       # a centre of its own per dimension
    q = (x[rng.integers(0, n, nq)] + rng.normal(0, 0.5, (nq, d))).astype(np.float32)
    q[0] += 5.0                                                                       # outside the rows' range
    ix = _index(vsk, dev, x)
    before = dev.stats()["reranked_rows"]
    got = ix.batchSearch(q, k)
    assert dev.stats()["reranked_rows"] > before
    assert_topk_parity(*got, *cpu_oracle.flat_search(oracle.MANHATTAN, q, x, k))
    ix.add(x[:100] + 40.0)                                                            # a wider range: the grid is made again
    assert_topk_parity(*ix.batchSearch(q, k), *cpu_oracle.flat_search(oracle.MANHATTAN, q, np.concatenate([x, x[:100] + 40.0]), k))


@pytest.mark.parametrize("masks", ["few", "many"])
def test_filters(vsk, dev, cpu_oracle, masks):
    """Few distinct masks: a row list per group of queries; many: one pass with the masks tested on listed rows."""
    rng = np.random.default_rng(9)
    n, d, nq = 60_000, 32, 300
    x = rng.uniform(-1, 1, (n, d)).astype(np.float32)
    q = rng.uniform(-1, 1, (nq, d)).astype(np.float32)
    rm = rng.integers(0, 2 ** 64, n, dtype=np.uint64)
    if masks == "few":
        qm = np.uint64(1) << rng.integers(0, 4, nq).astype(np.uint64)
    else:
        qm = rng.integers(1, 2 ** 64, nq, dtype=np.uint64)
        qm[:5] = 1 << 7
    got = _index(vsk, dev, x, rm).batchSearch(q, 20, qm)
    assert_topk_parity(*got, *cpu_oracle.flat_search(oracle.MANHATTAN, q, x, 20, rm, qm))


def test_outliers_ties_and_non_finite_values(vsk, dev, cpu_oracle):
    rng = np.random.default_rng(10)
    n, d, nq = 30_000, 24, 64
    x = rng.uniform(-1, 1, (n, d)).astype(np.float32)
    q = rng.uniform(-1, 1, (nq, d)).astype(np.float32)
    wide = x.copy()
    wide[123] = 1e6                                       # the step is wider than every distance: all lists overflow
    ix = _index(vsk, dev, wide)
    for _ in range(2):
        assert_topk_parity(*ix.batchSearch(q, 10), *cpu_oracle.flat_search(oracle.MANHATTAN, q, wide, 10))
    same = np.repeat(x[:3], n // 3, axis=0)               # thousands of rows at every distance
    assert_topk_parity(*_index(vsk, dev, same).batchSearch(q, 10), *cpu_oracle.flat_search(oracle.MANHATTAN, q, same, 10))
    const = np.full((n, d), 0.25, np.float32)             # no range at all
    assert_topk_parity(*_index(vsk, dev, const).batchSearch(q, 10), *cpu_oracle.flat_search(oracle.MANHATTAN, q, const, 10))
    bad = q.copy()
    bad[5, 3], bad[40, 0] = np.nan, np.inf
    keep = [i for i in range(nq) if i not in (5, 40)]
    d_, i_ = _index(vsk, dev, x).batchSearch(bad, 10)
    rd, ri = cpu_oracle.flat_search(oracle.MANHATTAN, q, x, 10)
    assert_topk_parity(d_[keep], i_[keep], rd[keep], ri[keep])
    inf = x.copy()
    inf[7, 2] = np.inf                                    # no grid: the fp32 scan
    assert_topk_parity(*_index(vsk, dev, inf).batchSearch(q, 10), *cpu_oracle.flat_search(oracle.MANHATTAN, q, inf, 10))


def test_a_row_that_is_not_a_number_among_many(vsk, dev, cpu_oracle):
    """A warp of the byte conversion takes several rows (more than 18 944 in all), so the NaN row must outlast the rows after
    it.  Query 0's filter passes four rows and the NaN row only: the fp32 scan does not list that row, and neither may this."""
    rng = np.random.default_rng(31)
    n, d, nq, bad = 60_000, 24, 64, 20_000
    x = rng.uniform(-1, 1, (n, d)).astype(np.float32)
    x[bad, 5] = np.nan
    q = rng.uniform(-1, 1, (nq, d)).astype(np.float32)
    rm = rng.integers(1, 2 ** 62, n, dtype=np.uint64)
    qm = rng.integers(1, 2 ** 62, nq, dtype=np.uint64)          # every query a mask of its own: one pass, not grouped
    qm[0] = np.uint64(1) << np.uint64(63)
    rm[[100, 30_000, 45_000, 59_999, bad]] |= qm[0]
    ix = _index(vsk, dev, x, rm)
    got = ix.batchSearch(q, 10, qm)
    plain = ix.batchSearch(q, 10)
    dev.set_search_path(1)
    try:
        ref, ref_plain = ix.batchSearch(q, 10, qm), ix.batchSearch(q, 10)
    finally:
        dev.set_search_path(0)
        ix.close()
    assert sorted(ref[1][0].tolist()) == [-1] * 6 + [100, 30_000, 45_000, 59_999]
    assert np.array_equal(got[1], ref[1]) and np.array_equal(got[0], ref[0])
    assert np.array_equal(plain[1], ref_plain[1]) and np.array_equal(plain[0], ref_plain[0])


def test_one_filter_group_that_overflows_does_not_shut_out_the_others(vsk, dev):
    rng = np.random.default_rng(32)
    groups, n, d, per = 5, 100_000, 128, 400
    x = rng.uniform(-1, 1, (n, d)).astype(np.float32)
    rm = np.uint64(1) << (np.arange(n) % groups).astype(np.uint64)
    q = rng.uniform(-1, 1, (groups * per, d)).astype(np.float32)
    qm = np.uint64(1) << (np.arange(groups * per) // per).astype(np.uint64)
    late = np.arange(n - 75_000, n)
    x[late[rm[late] == 1]] = 0.01                                # 15 000 equal rows, nearest to all of group 0's queries
    q[: per // 2] = 0.0
    q[5, 3] = np.nan                                             # no evidence of anything
    ix = _index(vsk, dev, x, rm)
    dev.set_search_path(1)
    ref = ix.batchSearch(q, 10, qm)
    dev.set_search_path(0)
    for _ in range(3):
        before = dev.stats()["fallback_queries"]
        got, names = logged_launches(dev, lambda: ix.batchSearch(q, 10, qm))
        assert dev.stats()["fallback_queries"] - before >= per
        assert names.count("l1_dense") == groups                 # all groups took the byte filter, on every call
        keep = np.arange(len(q)) != 5
        assert np.array_equal(got[1][keep], ref[1][keep]) and np.array_equal(got[0][keep], ref[0][keep])
    ix.close()


def test_filter_groups_take_turns_on_two_lanes(vsk, dev):
    """Groups of different sizes, one that no row passes, one too small for the byte filter and one whose lists overflow, on both
    lanes of the context: the fp32 scan's results, and the same again."""
    rng = np.random.default_rng(36)
    n, d = 480_000, 256
    x = rng.uniform(-1, 1, (n, d)).astype(np.float32)
    rm = np.uint64(1) << rng.integers(0, 6, n).astype(np.uint64)
    sizes = [300, 240, 9, 80, 200, 66, 64]                       # the seventh group's bit is on no row
    qm = np.concatenate([np.full(m, 1 << g, np.uint64) for g, m in enumerate(sizes)])
    q = rng.uniform(-1, 1, (len(qm), d)).astype(np.float32)
    late = np.arange(400_000, n)
    x[late[rm[late] == 16]] = 0.02                               # 13 000 equal rows, nearest to some of the fifth group's queries
    q[630:660] = 0.0
    order = rng.permutation(len(qm))
    q, qm = np.ascontiguousarray(q[order]), np.ascontiguousarray(qm[order])
    ix = _index(vsk, dev, x, rm)
    dev.set_search_path(1)
    ref = ix.batchSearch(q, 20, qm)
    dev.set_search_path(0)
    for call in range(3):
        dev.timeline(True)
        dev.timeline_read()
        got = ix.batchSearch(q, 20, qm)
        lanes = {lane for lane, what, _ in dev.timeline_read() if what == "l1_scan"}
        dev.timeline(False)
        assert call == 0 or {int(v) for v in lanes} == {0, 1}    # (the first batch does not pay for the byte copy)
        assert np.array_equal(got[1], ref[1]) and np.array_equal(got[0], ref[0])
    assert np.all(got[1][qm == 64] == -1)
    ix.close()


def test_filter_groups_take_one_lane_where_two_have_no_room(vsk):
    """With less free memory than the second lane's row list takes (90 MB), the groups take the first lane in turn."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(41)
    n, d, per, k = 20_000_000, 4, 40, 10
    x = torch.empty((n, d), device="cuda").uniform_(-1.0, 1.0, generator=gen)
    q = torch.empty((2 * per, d), device="cuda").uniform_(-1.0, 1.0, generator=gen)
    rm = (torch.arange(n, device="cuda") & 1) + 1
    qm = torch.arange(2 * per, device="cuda") // per + 1
    filler = None
    try:
        found = []
        for tight in (False, True):
            dev = vsk.CUDAAcceleratorStrategy(0).initialize()
            try:
                ix = _index(vsk, dev, x, rm)
                for group in (slice(0, per), slice(per, 2 * per)):   # one group at a time: the first lane's buffers
                    ix.batchSearch(q[group], k, qm[group])
                if tight:
                    filler = torch.empty(torch.cuda.mem_get_info()[0] - (72 << 20), dtype=torch.uint8, device="cuda")
                dev.timeline(True)
                dev.timeline_read()
                found.append(ix.batchSearch(q, k, qm))
                found[-1] += ({int(lane) for lane, _, _ in dev.timeline_read()},)
                dev.timeline(False)
                ix.close()
            finally:
                dev.close()
    finally:
        del filler
        torch.cuda.empty_cache()
    (d0, i0, lanes0), (d1, i1, _) = found
    assert lanes0 == {0, 1}
    assert torch.equal(i0, i1) and torch.equal(d0, d1) and bool((i1[:per] % 2 == 0).all()) and bool((i1[per:] % 2 == 1).all())


def test_more_filter_groups_than_are_counted_in_one_pass(vsk, dev, cpu_oracle):
    """105 distinct masks of two bits: the groups' rows are counted group by group, on one lane."""
    rng = np.random.default_rng(37)
    n, d, per, k = 60_000, 256, 100, 10                          # 1.1e9 steps a group: the byte filter pays
    x = rng.uniform(-1, 1, (n, d)).astype(np.float32)
    rm = rng.integers(0, 2 ** 15, n, dtype=np.uint64)
    masks = np.array([(1 << a) | (1 << b) for a in range(15) for b in range(a)], np.uint64)
    qm = rng.permutation(np.repeat(masks, per))
    q = rng.uniform(-1, 1, (len(qm), d)).astype(np.float32)
    ix = _index(vsk, dev, x, rm)
    dev.set_search_path(1)
    ref = ix.batchSearch(q, k, qm)
    dev.set_search_path(0)
    got, names = logged_launches(dev, lambda: ix.batchSearch(q, k, qm))
    ix.close()
    assert names.count("l1_dense") == len(masks)
    assert np.array_equal(got[1], ref[1]) and np.array_equal(got[0], ref[0])
    some = rng.choice(len(qm), 64, replace=False)
    assert_topk_parity(got[0][some], got[1][some], *cpu_oracle.flat_search(oracle.MANHATTAN, q[some], x, k, rm, qm[some]))


def test_only_rows_that_are_re_scored_are_counted(vsk, dev):
    """The k rows kept from chunk to chunk carry their exact values already."""
    rng = np.random.default_rng(33)
    n, d, nq, k = 40_000, 32, 64, 1_000
    ix = _index(vsk, dev, rng.uniform(-1, 1, (n, d)).astype(np.float32))
    q = rng.uniform(-1, 1, (nq, d)).astype(np.float32)
    before = dev.stats()
    _, names = logged_launches(dev, lambda: ix.batchSearch(q, k))
    after = dev.stats()
    counted, chunks = after["reranked_rows"] - before["reranked_rows"], names.count("l1_scan")
    assert chunks > 1 and after["fallback_queries"] == before["fallback_queries"]
    # a chunk adds 0.65 of the rows seen before it, and so lists about 0.65 k rows a query: less than the k it finds kept
    assert 0 < counted < nq * k * chunks
    ix.close()


def test_the_widest_rows_of_the_path(vsk, dev):
    """A query of 12 288 dimensions fills the 48 KB of the re-scoring kernel."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(35)
    x = torch.empty((16_384, 12_288), device="cuda").uniform_(-1.0, 1.0, generator=gen)
    q = torch.empty((192, 12_288), device="cuda").uniform_(-1.0, 1.0, generator=gen)
    ix = _index(vsk, dev, x)
    (gd, gi), names = logged_launches(dev, lambda: ix.batchSearch(q, 10))
    assert "l1_rescore" in names
    dev.set_search_path(1)
    rd, ri = ix.batchSearch(q, 10)
    dev.set_search_path(0)
    assert torch.equal(gi, ri) and torch.equal(gd, rd)
    ix.close()


def test_the_byte_copy_is_made_when_it_pays(vsk, dev):
    """Adding and searching in turn keeps to the fp32 tile for batches that would not pay for the copy; so do batches that are
    too small to gain from a copy that exists, and first batches over many rows.  Batches on rows that stay as they are pay for
    it together."""
    rng = np.random.default_rng(34)
    n, d, k = 60_000, 256, 10
    x = rng.uniform(-1, 1, (n, d)).astype(np.float32)
    q = rng.uniform(-1, 1, (900, d)).astype(np.float32)
    ix = _index(vsk, dev, x)

    def filtered(nq, index=None):
        index = index or ix
        dev.set_search_path(1)
        ref = index.batchSearch(q[:nq], k)
        dev.set_search_path(0)
        got, names = logged_launches(dev, lambda: index.batchSearch(q[:nq], k))
        assert np.array_equal(got[1], ref[1]) and np.array_equal(got[0], ref[0])
        return "l1_scan" in names

    assert filtered(32)                                          # 15 million elements: the first batch makes the copy
    assert not filtered(32) and filtered(80)                     # 0.5e9 and 1.2e9 steps
    for nq in (80, 256, 80, 256):
        ix.add(x[:50] * 0.9)
        assert not filtered(nq)
    # 1.1e10 steps and 110 per element are 826 queries over these rows
    assert [filtered(80) for _ in range(10)] == [False] * 7 + [True] * 3
    ix.add(x[:50] * 0.9)
    assert filtered(900)
    ix.close()
    wide = _index(vsk, dev, np.concatenate([x, x[:10_000] + 0.1]))   # 17.9 million elements, 724 queries
    assert [filtered(m, wide) for m in (80, 600, 80)] == [False, False, True]
    wide.close()
