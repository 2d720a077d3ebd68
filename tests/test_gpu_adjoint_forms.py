"""The three forms of the adjoint's backward sweep -- outside values stored and
the posteriors in a kernel of their own; posteriors in the sweep from kept
forward states; from recomputed ones -- give the same gradients and per-cell
values bit for bit: the same arithmetic per cell, and gradient sums over the
same runs of lines in the same order.  Sizes: one and several strips, partial
last strips, one-position queries and profiles, lines that make fewer than eight
runs, one line more or less than a multiple of eight runs, several 32-line
chunks a run."""
import numpy as np
import pytest

from comer2_b200 import synth as S

pytestmark = pytest.mark.gpu

THETA = np.array([0.05, -0.1, 0.02, 0.0, 0.1, -0.05, 0.03])


@pytest.mark.parametrize("qlens,dlens", [
    ((1, 32, 33, 70), (1, 9, 32, 33, 34, 97, 98)),
    ((31, 64, 65, 130), (1, 2, 224, 225, 226, 290, 411)),
])
def test_backward_forms_agree(params, qlens, dlens):
    from comer2_b200.native import Handle
    rng = np.random.default_rng(31)
    Q = S.random_profiles(rng, list(qlens))
    db = S.random_profiles(rng, list(dlens))
    qof, prof = (x.ravel().astype(np.int32) for x in np.mgrid[0:len(qlens), 0:len(dlens)])
    wss, wcv = params.ssswgt, params.cvswgt
    fbytes = 640 * sum((qlens[q] + 31) // 32 * (dlens[p] + 31) for q, p in zip(qof, prof))
    one_cta = 4 * (max(dlens) + 31) * 640
    margin = 64 << 10
    assert fbytes > one_cta + margin

    def run(limit):
        h = Handle(params, 0)
        h.upload_db(db)
        h.set_query_batch(Q)
        if limit:
            h.set_memory_limit(limit)
        z = h.logz_fwd_batch(qof, prof, THETA, wss, wcv)
        g = h.logz_bwd()
        cells = [h.logz_cells(k, int(dlens[p])) for k, p in enumerate(prof)]
        use = h.memory_use()
        assert np.array_equal(g, h.logz_bwd())     # again on the same forward sweep
        h.close()
        return z, g, cells, use

    out = run(0)
    kept = run(1 << 40)
    assert out[3] - kept[3] >= fbytes              # the outside values were stored without a limit only
    recomp = run(kept[3] - fbytes + one_cta + margin)
    assert recomp[3] <= kept[3] - fbytes + one_cta + margin
    for other in (kept, recomp):
        assert np.array_equal(out[0], other[0])
        assert np.array_equal(out[1], other[1])
        for (a0, b0), (a1, b1) in zip(out[2], other[2]):
            assert np.array_equal(a0, a1) and np.array_equal(b0, b1)
