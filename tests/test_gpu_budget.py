"""Device memory budget (c2_set_device_memory_limit, the reference's
--dev-mem): a budget too small for the database is refused with
C2_ERR_NOMEM before any allocation beyond it; a budget that holds the
database but not the phase-2 scratch of all candidate pairs makes c2_search
run phase 2 in candidate groups, with the same hits, statistics and
alignments as the unbounded search, and the handle's device memory never
above the budget."""
import numpy as np
import pytest

from comer2_b200 import synth as S

pytestmark = pytest.mark.gpu


def _pair_scratch_bytes(Lq, L, Lmax):
    """The library's estimate of one candidate pair's phase-2 device bytes
    (pair_scratch_bytes in c2_host.cu)."""
    ns = (Lq + 31) // 32
    return (9 * Lq * L + 2 * 5 * 4 * ns * (L + 12) + 4 * ns * 2 + 2 * 4 * 32 * ns * (L + 31)
            + 2 * 5 * (Lq + Lmax + 1) + 4 * 641 + 512)


def _key(rec, buf):
    raw = bytes(buf)
    out = []
    for r in rec:
        o, L = int(r["aln_offset"]), int(r["alnlen"])
        out.append((int(r["profile"]), float(r["score"]), float(r["logE"]), float(r["lambda_"]), float(r["K"]),
                    int(r["beg"]), int(r["end"]), raw[o:o + 5 * (L + 1)]))
    return out


@pytest.mark.parametrize("mode", [0, 1])
def test_budget_groups_give_the_same_hits(params, mode):
    from comer2_b200.native import Handle
    w = S.config(4, seed=3, scale=0.0008)   # 1 x 3000 vs 40 profiles, 2 planted homologs
    h = Handle(params, 0)
    h.set_score_mode(mode)
    h.upload_db(w.db, total_positions=18_000_000, total_profiles=50_000)
    ref = _key(*h.search(w.queries[0], arrays=True))
    assert h.search_groups() == 1 and len(ref) >= 2
    h.close()
    h = Handle(params, 0)
    h.set_score_mode(mode)
    h.upload_db(w.db, total_positions=18_000_000, total_profiles=50_000)
    h.set_query(w.queries[0])
    h.run_phase1()
    h.sync()
    base = h.memory_use()
    # room for the phase-2 scratch of the longest hit's pair and a little
    # more, so that the candidates go in several groups
    Lq = int(w.queries[0].lengths[0])
    longest = max(int(w.db.lengths[x[0]]) for x in ref)
    limit = base + (2 << 20) + int(1.3 * _pair_scratch_bytes(Lq, longest, int(w.db.lengths.max())) / 0.97)
    h.set_memory_limit(limit)
    got = _key(*h.search(w.queries[0], arrays=True))
    assert h.search_groups() >= 2
    assert h.memory_use() <= limit
    assert got == ref
    h.close()


def test_budget_below_the_database_is_refused(params):
    from comer2_b200.native import C2Error, Handle
    w = S.config(1, seed=4, scale=0.002)
    h = Handle(params, 0)
    h.set_memory_limit(h.memory_use() + 1 * 2**20)
    with pytest.raises(C2Error, match="C2_ERR_NOMEM"):
        h.upload_db(w.db)
    assert h.memory_use() <= h.memory_use() + 2**20
    h.set_memory_limit(0)
    h.upload_db(w.db)
    assert len(h.search(w.queries[0])) >= 1
    h.close()


@pytest.mark.parametrize("staged", [True, False])
@pytest.mark.parametrize("mode", [0, 1])
def test_split_scratch_gives_way(params, mode, staged):
    """The boundary rows of phase 1's split pairs (40 bytes a db column; with
    few pairs all are split) are not needed after it: under a limit that leaves
    phase 2 what it needs without them, the stages run, one by one and in a
    batch, within the limit and with the same hits."""
    from comer2_b200.native import Handle
    rng = np.random.default_rng(21)
    q = S.random_profiles(rng, [300])
    db = S.concat([S.planted_homolog(rng, q, 400, seg_lo=90, seg_hi=140) for _ in range(4)] +
                  [S.random_profiles(rng, [400] * 40)])
    rows = 40 * db.npositions

    def handle():
        h = Handle(params, 0)
        h.set_score_mode(mode)
        h.upload_db(db)
        return h

    def stages(h):
        h.set_query(q)
        h.run_phase1()
        use = h.memory_use()
        h.run_finalize()
        h.run_stats()
        return use, h.hits_arrays(h.run_map())

    h = handle()
    after1, (rec, buf) = stages(h)
    full = h.memory_use()
    assert len(rec) >= 4
    h.close()
    limit = full - rows + (64 << 10)
    h = handle()
    h.set_memory_limit(limit)
    if staged:
        use, got = stages(h)
        assert use == after1                   # the rows were there, and in phase 2's way
    else:
        got = h.search_batch(q, 1)[0]
    assert got[0].tobytes() == rec.tobytes() and np.array_equal(got[1], buf)
    assert h.memory_use() <= limit
    h.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_batch_under_a_limit_goes_in_groups(params, mode):
    """c2_search_batch runs a query whose candidates do not fit the limit at
    once in groups, as c2_search does, and the others as before."""
    from comer2_b200.native import Handle
    rng = np.random.default_rng(22)
    qs = S.random_profiles(rng, [300, 40])
    db = S.concat([S.planted_homolog(rng, qs.profile(0), 400, seg_lo=90, seg_hi=140) for _ in range(12)] +
                  [S.random_profiles(rng, [300] * 20)])

    def handle(limit):
        h = Handle(params, 0)
        h.set_score_mode(mode)
        h.upload_db(db)
        h.set_memory_limit(limit)
        return h

    h = handle(0)
    h.set_query(qs.profile(0))
    h.run_phase1()
    h.sync()
    base = h.memory_use()
    want = [_key(*h.search(qs.profile(k), arrays=True)) for k in range(2)]
    full = h.memory_use()
    assert len(want[0]) >= 12
    h.close()
    limit = base + (full - base) // 2
    h = handle(limit)
    got = [_key(*r) for r in h.search_batch(qs, 1)]
    assert got == want
    assert h.memory_use() <= limit
    got = h.search_batch(qs.profile(0), 1)
    assert h.search_groups() >= 2 and _key(*got[0]) == want[0]
    h.close()
