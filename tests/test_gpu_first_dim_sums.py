"""The external products' own sum over the giant steps: both of its kernels
(one ciphertext per CTA from 149 ciphertexts on a B200, a CTA per prime below),
one accumulator (N1 = 128, 256) and two (N1 = 64), and the first-dimension
results read back after each.  Word for word against the oracle."""
import numpy as np
import pytest

import kspir_b200 as kb
from kspir_b200 import serving
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r,N1,n", [(1, 64, 1), (1, 256, 1), (2, 64, 2), (16, 64, 10), (16, 128, 9), (16, 128, 10)])
def test_results_and_answers(r, N1, n):
    db = po.gen_db(501, r, N1)
    keys = po.gen_client(510, r, N1)
    q = serving.random_queries(np.random.default_rng(r * N1 + n), n)
    with kb.Context(r, N1, max_clients=1, max_inflight=max(n, 2)) as ctx:
        ctx.upload_db(db)
        ctx.upload_perms(keys["perms"])
        ctx.upload_client(0, keys["baby"], keys["giant"], keys["packing"], keys["rgsw"])
        got = ctx.answer_batch(np.zeros(n, np.int32), q)
        result = ctx.fetch_stage(kb.STAGE_RESULT, slot=n - 1).reshape(-1)
        staged, _ = ctx.matrix_vector_mul(0, q[n - 1])
        assert np.array_equal(result, staged)
        assert np.array_equal(ctx.fetch_stage(kb.STAGE_RESULT).reshape(-1), result)
        for i in {0, n - 1}:
            assert np.array_equal(got[i], po.answer(db, r, N1, dict(keys, query=q[i]))), i
