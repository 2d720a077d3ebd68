"""Handles of one process used from several threads at once: what they share
(the kernels' attributes, the pinned memory that handles borrow) must not let one
thread's call disturb another's.  Each result equals the same call's alone."""
import copy
import threading

import numpy as np
import pytest

from comer2_b200 import synth as S

pytestmark = pytest.mark.gpu


def _in_threads(fns, repeat):
    """Every function repeated in a thread of its own; their results, or the first error."""
    res, err = [[] for _ in fns], []

    def body(i):
        try:
            for _ in range(repeat):
                res[i].append(fns[i]())
        except BaseException as e:   # noqa: BLE001 (re-raised below)
            err.append(e)

    th = [threading.Thread(target=body, args=(i,)) for i in range(len(fns))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    if err:
        raise err[0]
    return res


@pytest.mark.parametrize("mode", [0, 1])
def test_searches_with_few_and_many_hits(params, mode):
    """The later stages' launch shapes depend on the number of hits: a search
    with one or two beside searches with many, over and over."""
    from comer2_b200.native import Handle
    rng = np.random.default_rng(5)
    sets = []
    for nhom in (1, 8, 40):
        q = S.random_profiles(rng, [70])
        parts = [S.planted_homolog(rng, q, 90, seg_lo=50, seg_hi=68) for _ in range(nhom)]
        sets.append((q, S.concat(parts + [S.random_profiles(rng, [60] * 20)])))
    hs, alone = [], []
    for q, db in sets:
        h = Handle(params, 0)
        h.set_score_mode(mode)
        h.upload_db(db)
        hs.append(h)
        alone.append(h.search(q, arrays=True))
    assert 0 < len(alone[0][0]) < len(alone[2][0])
    got = _in_threads([lambda h=h, q=q: h.search(q, arrays=True) for h, (q, _) in zip(hs, sets)], 60)
    for (ra, ba), runs in zip(alone, got):
        for rb, bb in runs:
            assert len(ra) == len(rb)
            for name in ra.dtype.names:
                assert np.array_equal(ra[name], rb[name]), name
            assert bytes(ba[:len(bb)]) == bytes(bb[:len(ba)])
    for h in hs:
        h.close()


def test_query_batches_and_many_handles(params):
    """Query batches packed at the same time (one gets the pinned block), in
    more handles than there are pinned slots."""
    from comer2_b200.native import Handle
    rng = np.random.default_rng(6)
    db = S.random_profiles(rng, [40, 61])
    small, large = S.random_profiles(rng, [33, 50]), S.random_profiles(rng, [500] * 8)
    theta = np.zeros(7)
    hs = []
    for _ in range(18):
        h = Handle(params, 0)
        h.upload_db(db)
        hs.append(h)

    def call(h, qs):
        h.set_query_batch(qs)
        n = qs.nprofiles
        z = h.logz_fwd_batch(np.arange(n, dtype=np.int32), np.arange(n, dtype=np.int32) % 2, theta, 1.0, 1.0)
        return z, h.logz_bwd()

    want = [call(hs[0], qs) for qs in (small, large)]
    for h in hs:                                   # every slot in use, then beyond
        assert all(np.array_equal(a, b) for a, b in zip(call(h, small), want[0]))
    got = _in_threads([lambda h=h, i=i: call(h, (small, large)[i % 2]) for i, h in enumerate(hs[-4:])], 10)
    for i, runs in enumerate(got):
        for z, g in runs:
            assert np.array_equal(z, want[i % 2][0]) and np.array_equal(g, want[i % 2][1])
    for h in hs:
        h.close()


@pytest.mark.parametrize("mode,cards", [(0, (93, 250)), (1, (93, 106))])
def test_context_vector_maps_of_different_sizes(params, mode, cards):
    """Handles whose kernels want different amounts of shared memory (the CV
    map's size), over and over in two threads."""
    from comer2_b200.native import Handle
    rng = np.random.default_rng(12)
    q = S.random_profiles(rng, [70])
    db = S.concat([S.planted_homolog(rng, q, 90, seg_lo=50, seg_hi=68), S.random_profiles(rng, [60] * 20)])
    hs, alone = [], []
    for card in cards:
        p = copy.deepcopy(params)
        n = card - len(p.cvs2s_keys)
        p.cvs2s_keys = np.concatenate([p.cvs2s_keys, p.cvs2s_keys[-1] + 0.5 * np.arange(1, n + 1)])
        p.cvs2s_values = np.concatenate([p.cvs2s_values, np.full(n, p.cvs2s_values[-1])])
        h = Handle(p, 0)
        h.set_score_mode(mode)
        h.upload_db(db)
        hs.append(h)
        alone.append(h.search(q, arrays=True))
        assert len(alone[-1][0]) >= 1

    def body(h):
        def run():
            h.set_query(q)
            for _ in range(20):
                h.run_phase1()
            h.phase1()
            return h.search(q, arrays=True)
        return run

    got = _in_threads([body(h) for h in hs], 150)
    for (ra, ba), runs in zip(alone, got):
        for rb, bb in runs:
            assert ra.tobytes() == rb.tobytes() and bytes(ba) == bytes(bb)
    for h in hs:
        h.close()
