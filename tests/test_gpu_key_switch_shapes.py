"""The baby-step kernel's two shapes (one component per CTA for a single query,
both for batches) on the edges of their dispatch, for each N1, with the
permutation matrix of the ring and with other in-range permutations (the
digits' gather follows the caller's, the b terms the ring's).  Word for word
against the oracle."""
import numpy as np
import pytest

import kspir_b200 as kb
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
N = po.N


@pytest.mark.parametrize("N1", [64, 128, 256])
@pytest.mark.parametrize("perms", ["ring", "other"])
def test_batches_of_one_two_and_three(N1, perms):
    r = 2
    db = po.gen_db(301, r, N1)
    clients = [po.gen_client(310 + i, r, N1) for i in range(2)]
    rng = np.random.default_rng(N1)
    if perms == "other":
        other = rng.integers(0, N, size=np.shape(clients[0]["perms"])).astype(np.int32)
        for c in clients:
            c["perms"] = other
    q = np.empty((3, 4 * N), np.uint64)
    q[:, :2 * N] = rng.integers(0, po.CRTMOD, size=(3, 2 * N), dtype=np.uint64)
    q[:, 2 * N:] = rng.integers(0, po.BSMOD, size=(3, 2 * N), dtype=np.uint64)
    q[2, :] = 0
    cl = np.array([0, 1, 0], np.int32)
    want = [po.answer(db, r, N1, dict(clients[cl[i]], query=q[i])) for i in range(3)]
    with kb.Context(r, N1, max_clients=2, max_inflight=3) as ctx:
        ctx.upload_db(db)
        ctx.upload_perms(clients[0]["perms"])
        for i, c in enumerate(clients):
            ctx.upload_client(i, c["baby"], c["giant"], c["packing"], c["rgsw"])
        for n in (1, 2, 3):
            got = ctx.answer_batch(cl[:n], q[:n])
            for i in range(n):
                assert (got[i] == want[i]).all(), (n, i)
        assert (ctx.answer(1, q[1]) == want[1]).all()
