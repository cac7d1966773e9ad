"""Batches of more than 32 queries whose last tile of the tensor-core scan is a
smaller one: both sides of each step of its rule (tails of 4, 8 and 16 queries,
and one of 17, which stays a tile of 32).  Word for word against the answers of
the queries by themselves, the first and the last against the oracle."""
import numpy as np
import pytest

import kspir_b200 as kb
from kspir_b200 import serving
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
R, N1, MMA32 = 2, 128, 4


@pytest.fixture(scope="module")
def server():
    db = po.gen_db(401, R, N1)
    keys = [po.gen_client(410 + i, R, N1) for i in range(2)]
    q = serving.random_queries(np.random.default_rng(11), 81)
    with kb.Context(R, N1, max_clients=2, max_inflight=81) as ctx:
        ctx.upload_db(db)
        ctx.upload_perms(keys[0]["perms"])
        for i, c in enumerate(keys):
            ctx.upload_client(i, c["baby"], c["giant"], c["packing"], c["rgsw"])
        want = [ctx.answer(i % 2, q[i]) for i in range(81)]
        for i in (0, 32, 80):
            assert np.array_equal(want[i], po.answer(db, R, N1, dict(keys[i % 2], query=q[i])))
        yield ctx, q, want


@pytest.mark.parametrize("n", [33, 36, 37, 40, 41, 48, 49, 65, 80, 81])
def test_tail_tiles(server, n):
    ctx, q, want = server
    ctx.set_scan_kind(n, MMA32)
    got = ctx.answer_batch(np.arange(n, dtype=np.int32) % 2, q[:n])
    for i in range(n):
        assert np.array_equal(got[i], want[i]), i
