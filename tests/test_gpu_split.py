"""Phase 1 with the longest pairs split into strip items: a database of many
short profiles and a few much longer than the mean (split pairs and whole pairs
in one launch), of few profiles (all split), and of equal ones (none split, or, with fewer pairs
a warp in the tensor-core form, all).
The strip kernel of the allocation-free entry point never splits and scores
with the same FP32 arithmetic, so the FP32 maxima and cells must be its bits;
the tensor-core form's maxima must lie within its rounding of them (1e-4
relative; a context-vector value at a bin edge moves one cell by one table
step, 0.05 allows for that in at most 2 % of the pairs, which needs sets of many
pairs: test_gpu_phase1.py has the tensor-core form on a dozen pairs).  That pairs
were split shows in the handle's device memory: their boundary rows, 40 bytes a
column, are allocated by the first phase 1 that splits any."""
import ctypes as C

import numpy as np
import pytest

from comer2_b200 import synth as S

pytestmark = pytest.mark.gpu

LENGTHS = {
    "mixed": [1, 2, 31, 32, 33, 700, 1999, 2000] + [20 + i % 41 for i in range(6000)],
    "few": [7, 64, 65, 300, 1001],
    "equal": [50] * 4000,
}


@pytest.mark.parametrize("lq", [32, 33, 64, 65, 129, 200])
@pytest.mark.parametrize("which", sorted(LENGTHS))
def test_split_pairs_match_whole_pairs(params, which, lq):
    import torch
    from comer2_b200.native import Handle
    rng = np.random.default_rng(lq)
    db = S.random_profiles(rng, LENGTHS[which])
    q = S.random_profiles(rng, [lq])
    h = Handle(params, 0)
    h.upload_db(db)
    h.set_query(q)
    n = db.nprofiles
    d_best = torch.full((n,), -1.0, dtype=torch.float32, device="cuda:0")
    d_coords = torch.full((n,), -1, dtype=torch.int32, device="cuda:0")
    torch.cuda.synchronize()
    h._ck(h.lib.c2_run_phase1_static(h._h, C.c_void_p(d_best.data_ptr()), C.c_void_p(d_coords.data_ptr())), "static")
    h.sync()
    ref = d_best.cpu().numpy()
    use = h.memory_use()
    # (of the mixed set the three pairs above the mean time per warp)
    split = {"mixed": 700 + 1999 + 2000, "few": sum(LENGTHS["few"]), "equal": 0}[which] if lq > 64 else 0
    for _ in range(2):   # the second run reuses the split pairs' scratch
        h.run_phase1()
        best, coords = h.phase1()
        assert np.array_equal(best.view(np.uint32), ref.view(np.uint32))
        assert np.array_equal(coords, d_coords.cpu().numpy().view(np.uint32))
        assert (h.memory_use() > use) == (split > 0) and h.memory_use() - use >= 40 * split
    if n >= 1000:
        h.set_score_mode(1)
        for _ in range(2):
            h.run_phase1()
            best, _ = h.phase1()
            d = np.abs(best - ref)
            assert (d <= 1e-4 * np.maximum(1.0, ref) + 0.05).all()
            assert (d <= 1e-4 * np.maximum(1.0, ref)).mean() >= 0.98
    h.close()
