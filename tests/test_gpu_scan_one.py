"""The tensor-core database scan of one query: that the answers meant to run on it
do, and their words.  Eight answers are issued on four streams that a sleeping
kernel holds up, so that how many others each finds in flight is known: none and
one for the first two (CUDA cores), two or three for the rest (tensor cores from 64
database rows on).  A tile chosen for n = 1 means the same scan, on every stream and at
any number of rows.  Word for word against the same queries alone and the oracle,
also with every database half at 2^32 - 1 (sums that wrap modulo 2^64)."""
import time

import numpy as np
import pytest
import torch

import kspir_b200 as kb
from kspir_b200 import serving
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
N = po.N
N1, ANSWERS = 128, 8   # one per workspace slot of the single answers


def context(r, db, keys):
    ctx = kb.Context(r, N1, max_clients=1, max_inflight=8)
    ctx.upload_db(db)
    ctx.upload_perms(keys["perms"])
    ctx.upload_client(0, keys["baby"], keys["giant"], keys["packing"], keys["rgsw"])
    return ctx


def database(r, fill):
    return np.full(r * N * N // 2, np.uint64(0xFFFFFFFFFFFFFFFF)) if fill == "ones" else po.gen_db(701, r, N1)


def issue(ctx, q):
    """Responses of the queries issued side by side, and each one's scan variant."""
    d_q = torch.from_numpy(q.view(np.int64)).cuda()
    d_r = torch.zeros((ANSWERS, 2 * N), dtype=torch.int64, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    for s in streams:
        with torch.cuda.stream(s):
            torch.cuda._sleep(200_000_000)   # a tenth of a second
    for i in range(ANSWERS):
        ctx.answer_device(0, d_q[i].data_ptr(), d_r[i].data_ptr(), streams[i % 4].cuda_stream)
    kinds = [ctx.slot_scan_kind(i) for i in range(ANSWERS)]
    ctx.sync()
    return d_r.cpu().numpy().view(np.uint64), kinds


@pytest.mark.parametrize("r,fill", [(2, "words"), (4, "words"), (4, "ones"), (8, "words"), (16, "ones")])
def test_answers_beside_others(r, fill):
    db, keys = database(r, fill), po.gen_client(710, r, N1)
    q = serving.random_queries(np.random.default_rng(r), ANSWERS)
    q[3] = 0
    with context(r, db, keys) as ctx:
        alone = [ctx.answer(0, q[i]) for i in range(ANSWERS)]
        assert [ctx.slot_scan_kind(i) for i in range(ANSWERS)] == [kb.SCAN_CUDA] * ANSWERS
        got, kinds = issue(ctx, q)
        beside = kb.SCAN_ONE if r * (N // 2 // N1) >= 64 else kb.SCAN_CUDA
        assert kinds == [kb.SCAN_CUDA] * 2 + [beside] * (ANSWERS - 2)
        for i in range(ANSWERS):
            assert np.array_equal(got[i], alone[i]), i
        for i in (2, 3, 7):
            assert np.array_equal(got[i], po.answer(db, r, N1, dict(keys, query=q[i]))), i


@pytest.mark.parametrize("r,kind", [(1, kb.SCAN_MMA4), (2, kb.SCAN_MMA8), (4, kb.SCAN_MMA16), (4, kb.SCAN_MMA32)])
def test_tile_chosen_for_one_query(r, kind):
    db, keys = database(r, "words"), po.gen_client(720, r, N1)
    q = serving.random_queries(np.random.default_rng(20 + r), ANSWERS)
    want = [po.answer(db, r, N1, dict(keys, query=x)) for x in q]
    with context(r, db, keys) as ctx:
        ctx.set_scan_kind(1, kind)
        assert ctx.scan_kind(1) == kind
        for _ in range(3):
            got, kinds = issue(ctx, q)
            assert kinds == [kb.SCAN_ONE] * ANSWERS
            for i in range(ANSWERS):
                assert np.array_equal(got[i], want[i]), i
        assert np.array_equal(ctx.answer(0, q[0]), want[0])   # slot 0 again
        scan = ctx.fetch_stage(kb.STAGE_SCAN)
        assert np.array_equal(ctx.answer_batch(np.zeros(1, np.int32), q[:1])[0], want[0])
        assert np.array_equal(ctx.fetch_stage(kb.STAGE_SCAN), scan)
        ctx.set_scan_kind(1, kb.SCAN_CUDA)
        assert np.array_equal(ctx.answer_batch(np.zeros(1, np.int32), q[:1])[0], want[0])
        assert np.array_equal(ctx.fetch_stage(kb.STAGE_SCAN), scan)


def test_tuning_for_one_query_leaves_the_rule_beside_others():
    r = 4
    db, keys = database(r, "words"), po.gen_client(730, r, N1)
    q = serving.random_queries(np.random.default_rng(30), ANSWERS)
    with context(r, db, keys) as ctx:
        alone = [ctx.answer(0, q[i]) for i in range(ANSWERS)]
        tuned, _ = ctx.tune_batch(1)
        assert ctx.scan_kind(1) == tuned
        ctx.answer(0, q[0])
        assert ctx.slot_scan_kind(0) == (kb.SCAN_CUDA if tuned == kb.SCAN_CUDA else kb.SCAN_ONE)
        for i in range(1, ANSWERS):   # slot 0 comes next again
            ctx.answer(0, q[i])
        for choose, beside in ((None, kb.SCAN_ONE), (kb.SCAN_CUDA, kb.SCAN_CUDA), (-1, kb.SCAN_ONE)):
            if choose is not None:
                ctx.set_scan_kind(1, choose)
            got, kinds = issue(ctx, q)
            assert kinds[2:] == [beside] * (ANSWERS - 2), choose
            for i in range(ANSWERS):
                assert np.array_equal(got[i], alone[i]), i


@pytest.mark.parametrize("skip", [0, 3, 9])   # in the first lap of the ring of four tiles, its end, the third
def test_wait_runs_out_after_the_callers_limit(skip):
    r = 4
    db, keys = database(r, "words"), po.gen_client(740, r, N1)
    want = po.answer(db, r, N1, keys)
    with context(r, db, keys) as ctx:
        ctx.set_scan_kind(1, kb.SCAN_MMA4)
        assert np.array_equal(ctx.answer(0, keys["query"]), want)
        ctx.debug_scan_fault(wait_limit_ns=1_000_000, skip_item=skip)
        t0 = time.perf_counter()
        with pytest.raises(kb.KspirError) as e:
            ctx.answer(0, keys["query"])
        assert e.value.code == kb.native.ERR_TIMEOUT
        assert time.perf_counter() - t0 < 1.0   # not the default limit of two seconds
        for _ in range(ANSWERS):
            assert np.array_equal(ctx.answer(0, keys["query"]), want)
        ctx.debug_scan_fault()
        assert np.array_equal(ctx.answer(0, keys["query"]), want)
