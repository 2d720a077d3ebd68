"""Failure handling on the GPU without faulting it: the bounded waits between
the strips of one pair (phase 1's split pairs, the traceback, MAP and adjoint
sweeps) give up after the poll limit set with c2_set_wait_limit, the sweep
returns, and the call reports the device status (C2_ERR_DEVICE) instead of
hanging; the handle then serves the next call."""
import numpy as np
import pytest

from comer2_b200 import synth as S

pytestmark = pytest.mark.gpu

PHASE1 = "a wait in phase 1 timed out"
SWEEP = "a strip wait timed out"


def _strip_key(hits):
    return [(int(x["profile"]), round(float(x["score"]), 4), x["strings"][0]) for x in hits]


def test_traceback_sweep_wait_timeout(params):
    """One poll per wait from the finalisation on: strips started beside their
    predecessor give up at once in the traceback sweep (c2_run_finalize);
    c2_get_finalize and c2_run_stats report it."""
    from comer2_b200.native import C2Error, Handle
    w = S.config(1, seed=2, scale=0.003)   # 1 x 400 (13 strips) vs 300 profiles
    h = Handle(params, 0)
    h.upload_db(w.db)
    good = h.search(w.queries[0])
    assert len(good) > 0
    h.set_query(w.queries[0])
    h.run_phase1()
    h.phase1()
    h.set_wait_limit(1)
    n = h.run_finalize()
    assert n > 0
    with pytest.raises(C2Error, match=SWEEP):
        h.finalize(n)
    with pytest.raises(C2Error, match=SWEEP):
        h.run_stats()
    h.set_wait_limit(0)
    again = h.search(w.queries[0])
    assert _strip_key(again) == _strip_key(good)
    h.close()


def test_map_sweep_wait_timeout(params):
    """The same in the MAP forward-backward and MAP DP sweeps: phase 1,
    finalisation and statistics run with the default limit, MAP with one
    poll per wait; c2_get_hits reports the timeout."""
    from comer2_b200.native import C2Error, Handle
    w = S.config(1, seed=9, scale=0.003)
    h = Handle(params, 0)
    h.upload_db(w.db)
    h.set_query(w.queries[0])
    h.run_phase1()
    h.run_finalize()
    h.run_stats()
    h.set_wait_limit(1)
    n = h.run_map()
    assert n > 0
    with pytest.raises(C2Error, match=SWEEP):
        h.hits(n)
    h.set_wait_limit(0)
    assert len(h.search(w.queries[0])) == n
    h.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_phase1_wait_timeout(params, mode):
    """Phase 1 with one poll per wait: the strips of split pairs (with 300
    profiles, fewer than the warps, every pair is split) give up;
    c2_get_phase1 and a whole search report phase 1's wait."""
    from comer2_b200.native import C2Error, Handle
    w = S.config(1, seed=2, scale=0.003)
    h = Handle(params, 0)
    h.set_score_mode(mode)
    h.upload_db(w.db)
    h.set_query(w.queries[0])
    h.run_phase1()
    good = h.phase1()[0]
    h.set_wait_limit(1)
    h.run_phase1()
    with pytest.raises(C2Error, match=PHASE1):
        h.phase1()
    with pytest.raises(C2Error, match=PHASE1):
        h.search(w.queries[0])
    h.set_wait_limit(0)
    h.set_query(w.queries[0])
    h.run_phase1()
    assert np.array_equal(h.phase1()[0].view(np.uint32), good.view(np.uint32))
    h.close()


def test_adjoint_wait_timeout(params):
    """The adjoint's forward and backward sweeps: c2_logz_fwd / c2_logz_bwd
    report the wait, the next forward call starts clean."""
    from comer2_b200.native import C2Error, Handle
    rng = np.random.default_rng(4)
    db = S.random_profiles(rng, [900] * 8)
    q = S.random_profiles(rng, [300])
    h = Handle(params, 0)
    h.upload_db(db)
    h.set_query(q)
    pr = np.arange(8, dtype=np.int32)
    z, g = h.logz_fwd(pr, None, 1.0, 1.0), h.logz_bwd()
    h.set_wait_limit(1)
    with pytest.raises(C2Error, match=SWEEP):
        h.logz_fwd(pr, None, 1.0, 1.0)
    h.set_wait_limit(0)
    assert np.array_equal(h.logz_fwd(pr, None, 1.0, 1.0), z)
    h.set_wait_limit(1)
    with pytest.raises(C2Error, match=SWEEP):
        h.logz_bwd()
    h.set_wait_limit(0)
    assert np.array_equal(h.logz_fwd(pr, None, 1.0, 1.0), z)
    assert np.array_equal(h.logz_bwd(), g)
    h.close()


def test_candidates_of_a_timed_out_phase1_are_refused(params):
    """The maxima of a phase 1 whose wait gave up are no candidates: the
    finalisation reports the wait instead of working on them.  (With 300
    profiles, fewer than the warps, the strips of every pair are split.)"""
    from comer2_b200.native import C2Error, Handle
    w = S.config(1, seed=2, scale=0.003)
    h = Handle(params, 0)
    h.upload_db(w.db)
    h.set_query(w.queries[0])
    h.set_wait_limit(1)
    h.run_phase1()
    with pytest.raises(C2Error, match=PHASE1):
        h.run_finalize()
    h.close()


def test_adjoint_leaves_the_search_status(params):
    """A forward call of the adjoint between a timed-out phase 1 and its fetch
    does not clear phase 1's status; nor does a search's status fail it."""
    from comer2_b200.native import C2Error, Handle
    w = S.config(1, seed=2, scale=0.003)
    h = Handle(params, 0)
    h.upload_db(w.db)
    h.set_query(w.queries[0])
    pr = np.arange(4, dtype=np.int32)
    z = h.logz_fwd(pr, None, 1.0, 1.0)
    h.set_wait_limit(1)
    h.run_phase1()
    h.sync()
    h.set_wait_limit(0)
    assert np.array_equal(h.logz_fwd(pr, None, 1.0, 1.0), z)
    h.logz_bwd()
    with pytest.raises(C2Error, match=PHASE1):
        h.phase1()
    h.close()
