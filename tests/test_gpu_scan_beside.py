"""Single answers in flight beside others: their database scan runs on the tensor
cores (one query).  Row counts below, at and above one 32-row tile and several
units of slots per CTA, answers spread over streams without a wait in between.
Word for word against the same query alone, and the oracle."""
import numpy as np
import pytest
import torch

import kspir_b200 as kb
from kspir_b200 import serving
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
N = po.N


@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_answers_on_four_streams(r):
    N1, n = 128, 12
    db = po.gen_db(501, r, N1)
    keys = [po.gen_client(510 + i, r, N1) for i in range(2)]
    q = serving.random_queries(np.random.default_rng(r), n)
    q[n - 1] = 0
    q[n - 2, :2 * N], q[n - 2, 2 * N:] = po.CRTMOD - 1, po.BSMOD - 1
    with kb.Context(r, N1, max_clients=2, max_inflight=8) as ctx:
        ctx.upload_db(db)
        ctx.upload_perms(keys[0]["perms"])
        for i, c in enumerate(keys):
            ctx.upload_client(i, c["baby"], c["giant"], c["packing"], c["rgsw"])
        want = [ctx.answer(i % 2, q[i]) for i in range(n)]
        for i in (0, n - 2, n - 1):
            assert np.array_equal(want[i], po.answer(db, r, N1, dict(keys[i % 2], query=q[i])))
        d_q = torch.from_numpy(q.view(np.int64)).cuda()
        d_r = torch.zeros((n, 2 * N), dtype=torch.int64, device="cuda")
        streams = [torch.cuda.Stream() for _ in range(4)]
        torch.cuda.synchronize()
        for rep in range(3):
            for i in range(n):
                ctx.answer_device(i % 2, d_q[i].data_ptr(), d_r[i].data_ptr(), streams[i % 4].cuda_stream)
        ctx.sync()
        got = d_r.cpu().numpy().view(np.uint64)
        for i in range(n):
            assert np.array_equal(got[i], want[i]), i
