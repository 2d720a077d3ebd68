"""Context-vector scores beyond the range of integers: a determinant of 0 (its
logarithm -inf, the score +inf) and priors of billions take the map's last or
first value, in the FP32 kernels whose table index is clamped only (maps whose
keys sit at the table's ends) as in the strip kernel, which compares the keys,
and in the tensor-core form."""
import ctypes as C

import numpy as np
import pytest

from comer2_b200 import synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["det0", "prior-", "prior+"])
def test_scores_beyond_the_map(params, orc32, what):
    import torch
    from comer2_b200.native import Handle
    rng = np.random.default_rng(17)
    q = S.random_profiles(rng, [90])
    db = S.concat([S.planted_homolog(rng, q, 120, seg_lo=60, seg_hi=80), S.random_profiles(rng, [1, 40, 65, 200])])
    for ps in (q, db):
        if what == "det0":
            # (-1 + 1 + 1/kappa0)^2 - (0 + 1/kappa0)^2 = 0 in every cell
            ps.cv[...] = 0.0
            ps.cvnorm2[...] = -1.0
        else:
            ps.cvprior[...] = -2e9 if what == "prior-" else 2e9
    n = db.nprofiles
    h = Handle(params, 0)
    h.upload_db(db)
    h.set_query(q)
    b = torch.zeros(n, dtype=torch.float32, device="cuda:0")
    c = torch.zeros(n, dtype=torch.int32, device="cuda:0")
    torch.cuda.synchronize()
    h._ck(h.lib.c2_run_phase1_static(h._h, C.c_void_p(b.data_ptr()), C.c_void_p(c.data_ptr())), "static")
    h.sync()
    want = b.cpu().numpy()
    h.run_phase1()
    best, coords = h.phase1()
    assert np.array_equal(best.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(coords, c.cpu().numpy().view(np.uint32))
    qo = orc32.profile(q)
    for k in range(n):
        r = orc32.pair(qo, orc32.profile(db, k))["best"]
        assert abs(float(best[k]) - r) <= 1e-4 * max(1.0, abs(r)), k
    ncand = h.run_finalize()
    assert ncand >= 1
    sm, _ = h.pair_scores(0, int(db.lengths[0]))
    rs, _ = orc32.score_matrix(qo, orc32.profile(db, 0))
    assert np.abs(sm - rs).max() <= 5e-5          # test_gpu_phase1.py: the logarithms' difference
    h.set_score_mode(1)
    h.run_phase1()
    tc, _ = h.phase1()
    assert (np.abs(tc - want) <= 1e-4 * np.maximum(1.0, want)).all()
    h.close()
