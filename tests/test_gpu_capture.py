"""Stream capture.  Phase 1 allocates nothing and waits for nothing once its
operands are there, so it can be captured into a CUDA graph, on a handle's
first phase 1 of a query too; c2_set_query and c2_set_query_batch copy from
host memory that later calls use again, and refuse."""
import numpy as np
import pytest

from comer2_b200 import synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
@pytest.mark.parametrize("mode", [0, 1])
def test_phase1_captured(params, mode):
    import torch
    from comer2_b200.native import C2Error, Handle
    rng = np.random.default_rng(8)
    db = S.random_profiles(rng, [20, 64, 300, 1001])     # few pairs: split where nothing forbids it
    short, q, q2 = (S.random_profiles(rng, [n]) for n in (20, 200, 200))
    ref = Handle(params, 0)
    ref.set_score_mode(mode)
    ref.upload_db(db)
    want = []
    for x in (q, q2):
        ref.set_query(x)
        ref.run_phase1()
        want.append(ref.phase1())
    h = Handle(params, 0)
    h.set_score_mode(mode)
    h.upload_db(db)
    stream = torch.cuda.Stream()
    h.set_stream(stream.cuda_stream)
    h.set_query(short)
    h.run_phase1()                    # (packs the tensor-core operands of the database)
    h.set_score_mode(0)
    h.set_query(q)
    h.set_score_mode(mode)            # (and of a query set in the other mode)
    h.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        h.run_phase1()
    for x, (best, coords) in zip((q, q2), want):
        h.set_query(x)
        with torch.cuda.stream(stream):
            g.replay()
        b, c = h.phase1()
        assert np.array_equal(b.view(np.uint32), best.view(np.uint32)) and np.array_equal(c, coords)
    g2 = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g2, stream=stream):
        with pytest.raises(C2Error, match="capture"):
            h.set_query(q)
        with pytest.raises(C2Error, match="capture"):
            h.set_query_batch(q)
    h.set_query(q)
    h.run_phase1()
    assert np.array_equal(h.phase1()[0].view(np.uint32), want[0][0].view(np.uint32))
    h.set_stream(0)
    del g, g2
    h.close()
    ref.close()
