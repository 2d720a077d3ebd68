"""The caller's query arrays are free once c2_set_query / c2_set_query_batch has
returned, page-locked ones too, from which a copy is asynchronous: overwritten
at once, with an earlier phase 1 still queued on the handle's stream, they give
the bits of a call whose arrays stay."""
import ctypes as C

import numpy as np
import pytest

from comer2_b200 import synth as S

pytestmark = pytest.mark.gpu

FIELDS = ("bkg", "eno", "trn", "trg", "cv", "cvprior", "cvnorm2", "ss", "ssstate", "aa")


def _page_locked(ps):
    """A copy of the profiles in page-locked arrays, and what keeps them alive."""
    import copy
    import torch
    out, keep = copy.copy(ps), []
    for f in FIELDS:
        a = np.ascontiguousarray(getattr(ps, f))
        t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
        t.numpy()[...] = a
        keep.append(t)
        setattr(out, f, t.numpy())
    return out, keep


def _overwrite(ps):
    """Other valid values in place."""
    for f in FIELDS:
        a = getattr(ps, f)
        a[...] = a[::-1].copy() if f != "bkg" else 0.05
    ps.aa[...] = ord("A")
    ps.ssstate[...] = ord("C")
    ps.trn[...] = -1.0


def _database(rng, q, lens, others):
    parts = [S.planted_homolog(rng, q, L, seg_lo=min(60, int(q.lengths[0])), seg_hi=min(100, int(q.lengths[0])))
             for L in lens]
    return S.concat(parts + [S.random_profiles(rng, others)])


def _search_stages(h):
    h.run_phase1()
    best, coords = h.phase1()
    h.run_finalize()
    h.run_stats()
    rec, buf = h.hits_arrays(h.run_map())
    return best, coords, rec, buf


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("lq", [100, 330, 600, 1500, 5000])
def test_query_arrays_overwritten_after_set_query(params, mode, lq):
    from comer2_b200.native import Handle
    rng = np.random.default_rng(lq)
    q = S.random_profiles(rng, [lq])
    db = _database(rng, q, [120, 150, 200], [200] * 1500)
    busy = S.random_profiles(rng, [2000])
    h = Handle(params, 0)
    h.set_score_mode(mode)
    h.upload_db(db)
    h.set_query(q)
    want = _search_stages(h)
    assert len(want[2]) >= 3
    for _ in range(2):
        h.set_query(busy)
        h.run_phase1()               # milliseconds of work before the next query's copies
        pinned, keep = _page_locked(q)
        h.set_query(pinned)
        _overwrite(pinned)
        got = _search_stages(h)
        assert np.array_equal(got[0].view(np.uint32), want[0].view(np.uint32))
        assert np.array_equal(got[1], want[1])
        assert got[2].tobytes() == want[2].tobytes()
        assert np.array_equal(got[3], want[3])
        del keep
    h.close()


def test_many_queries_without_a_fetch(params):
    """Queries set one after the other with nothing but the allocation-free
    phase 1 and c2_sync between them."""
    import torch
    from comer2_b200.native import Handle
    rng = np.random.default_rng(3)
    qs = [S.random_profiles(rng, [int(n)]) for n in rng.integers(60, 200, 24)]
    db = S.random_profiles(rng, [150] * 600)
    n = db.nprofiles
    h = Handle(params, 0)
    h.upload_db(db)
    out = [(torch.zeros(n, dtype=torch.float32, device="cuda:0"), torch.zeros(n, dtype=torch.int32, device="cuda:0"))
           for _ in qs]
    torch.cuda.synchronize()
    want = []
    for q in qs:
        h.set_query(q)
        h.run_phase1()
        want.append(h.phase1()[0])
    for _ in range(2):
        for q, (b, c) in zip(qs, out):
            pinned, keep = _page_locked(q)
            h.set_query(pinned)
            _overwrite(pinned)
            for _ in range(3):
                h._ck(h.lib.c2_run_phase1_static(h._h, C.c_void_p(b.data_ptr()), C.c_void_p(c.data_ptr())), "static")
            del keep
        h.sync()
        for w, (b, _) in zip(want, out):
            assert np.array_equal(b.cpu().numpy().view(np.uint32), w.view(np.uint32))
    h.close()


@pytest.mark.parametrize("qlens", [(70, 90), (500,) * 40])
def test_query_arrays_overwritten_after_set_query_batch(params, qlens):
    from comer2_b200.native import Handle
    rng = np.random.default_rng(7)
    qs = S.random_profiles(rng, list(qlens))
    db = S.random_profiles(rng, [200] * 1500)
    busy = S.random_profiles(rng, [2000])
    n = len(qlens)
    qi, pr = np.arange(n, dtype=np.int32), np.arange(n, dtype=np.int32)
    h = Handle(params, 0)
    h.upload_db(db)

    def call():
        return h.logz_fwd_batch(qi, pr, np.full(7, 0.05), 1.0, 1.0), h.logz_bwd()

    h.set_query_batch(qs)
    want = call()
    h.set_query(busy)
    h.run_phase1()
    pinned, keep = _page_locked(qs)
    h.set_query_batch(pinned)
    _overwrite(pinned)
    got = call()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    del keep
    h.close()
