"""The first-dimension results of a batch of more ciphertexts than SMs, read back
after other calls have reused the scan output that their sums were left in: the
staged packing (slot 0), the staged external product of fewer ciphertexts (slot 0;
the others' results stay) and the scan tuning (every slot of the batch, here from
cipherbufs in the other layout than its last variant reads).  One accumulator
(N1 = 128) and two (N1 = 64).  Word for word against the results read straight after
the batch and against the staged first dimension."""
import numpy as np
import pytest

import kspir_b200 as kb
from kspir_b200 import serving
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
R, BATCH = 4, 38   # 152 ciphertexts, one of them per CTA on 148 SMs


@pytest.mark.parametrize("N1", [64, 128])
@pytest.mark.parametrize("between", ["packing", "external", "tune"])
def test_results_survive(N1, between):
    db = po.gen_db(601, R, N1)
    keys = po.gen_client(610, R, N1)
    q = serving.random_queries(np.random.default_rng(N1), BATCH)
    cl = np.zeros(BATCH, np.int32)
    with kb.Context(R, N1, max_clients=1, max_inflight=BATCH) as ctx:
        ctx.upload_db(db)
        ctx.upload_perms(keys["perms"])
        ctx.upload_client(0, keys["baby"], keys["giant"], keys["packing"], keys["rgsw"])
        first = ctx.matrix_vector_mul(0, q[0])[0]
        ctx.set_scan_kind(BATCH, kb.SCAN_CUDA)
        answers = ctx.answer_batch(cl, q)
        last = ctx.fetch_stage(kb.STAGE_RESULT, slot=BATCH - 1)
        if between == "packing":
            ctx.packing(0, ctx.fetch_stage(kb.STAGE_EXT).reshape(-1))
        elif between == "external":
            given = first[2 * po.N:4 * po.N]   # result 0 becomes the ciphertext passed in
            ctx.external_product(0, np.zeros(2 * po.N, np.uint64), given)
            first[:2 * po.N] = given
        else:
            ctx.tune_batch(BATCH)
        for _ in range(2):   # reading changes nothing
            assert np.array_equal(ctx.fetch_stage(kb.STAGE_RESULT).reshape(-1), first)
            assert np.array_equal(ctx.fetch_stage(kb.STAGE_RESULT, slot=BATCH - 1), last)
        assert np.array_equal(ctx.answer_batch(cl, q), answers)
        assert np.array_equal(answers[0], po.answer(db, R, N1, dict(keys, query=q[0])))
