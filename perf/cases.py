"""The work that is measured: what a server built on kspir_b200 has it do.

Each case goes through the package's public entry points on inputs made from a
seed: a raw database preprocessed on the device, client keys and queries of
uniform canonical words (what keys and queries under fresh randomness look
like).  Sizes are those of the repository's configurations, tests and
benchmark: r sub-databases (r = 16 is the 256 MB-record database, r = 64 the
1 GB one), N1 baby-step columns, and batch sizes from one query to 64.

Kinds of work:

* ``single``   one client's query answered from host buffers (Context.answer)
* ``overlap``  queries of several clients answered one by one on eight streams
  (Context.answer_device), as a server with several connections issues them
* ``batch``    n queries of several clients in one call (Context.answer_batch_device)
* ``hosted``   the same on host buffers, as a front end with the queries of a
  network poll calls it (Context.answer_batch)
* ``refresh``  a new raw database preprocessed on the device, then a query
  answered from it
* ``staged``   the three functions of the reference's interface one after
  another on host buffers, as a program written against the reference calls them
* ``clients``  the client side: n queries made and n responses decrypted

Every output is whole numbers (words modulo the ring's moduli): two builds
give the same words.
"""
from __future__ import annotations

import numpy as np
import torch

import kspir_b200 as kb

N = kb.N
STREAMS = 8


def listed():
    return [
        # the smallest call: one sub-database, where launches and latency are all
        dict(name="single_r1", kind="single", r=1, N1=128, n=1, clients=1),
        # the benchmark's query: 256 MB of records, one query at a time
        dict(name="single_256mb", kind="single", r=16, N1=128, n=1, clients=1),
        # the same from several connections at once (the benchmark's headline)
        dict(name="overlap_256mb", kind="overlap", r=16, N1=128, n=32, clients=8),
        # the reference's other baby-step split: more giant steps, fewer rotations
        dict(name="single_n64", kind="single", r=8, N1=64, n=1, clients=1),
        # the 1 GB database, one query at a time
        dict(name="single_1gb", kind="single", r=64, N1=128, n=1, clients=1),
        # a full batch of the benchmark, its scan tuned at start-up
        dict(name="batch64_256mb", kind="batch", r=16, N1=128, n=64, clients=16, tuned=True),
        # a batch as it happens to come: odd size, small database, nothing tuned
        dict(name="batch13_r4", kind="batch", r=4, N1=128, n=13, clients=5, tuned=False),
        # the benchmark's batch over the 1 GB database
        dict(name="batch32_1gb", kind="batch", r=64, N1=128, n=32, clients=16, tuned=True),
        # what one network poll brought in, from and to host buffers
        dict(name="hosted40_256mb", kind="hosted", r=16, N1=128, n=40, clients=12, tuned=False),
        # a database update
        dict(name="refresh_256mb", kind="refresh", r=16, N1=128, n=1, clients=1),
        # a program written against the reference's functions
        dict(name="staged_256mb", kind="staged", r=16, N1=128, n=1, clients=1),
        # load generation and test clients
        dict(name="clients_100", kind="clients", r=16, N1=128, n=100, clients=1),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["single", "overlap", "batch", "batch", "batch", "hosted", "refresh", "staged", "clients"])
    r = 1 << rng.randrange(0, 7)
    N1, n, clients = 128, 1, 1
    if kind in ("single", "staged"):
        N1 = rng.choice([64, 128, 128, 256])
        r = min(r, 64 if N1 == 128 else 16)
    elif kind == "overlap":
        r = min(r, 16)
        n = rng.randrange(2, 33)
        clients = rng.randrange(1, 9)
    elif kind in ("batch", "hosted"):
        n = _log_int(rng, 2, min(64, 1024 // r))
        clients = rng.randrange(1, min(n, 16) + 1)
    elif kind == "refresh":
        N1 = rng.choice([64, 128, 128, 256])
        r = min(r, 16)
    else:
        n = _log_int(rng, 1, 128)
        r = 1 << rng.randrange(1, 7)
    case = dict(kind=kind, r=r, N1=N1, n=n, clients=clients)
    if kind in ("batch", "hosted"):
        case["tuned"] = rng.random() < 0.5
    return case


# ---------------------------------------------------------------------------
# inputs

def _words(gen, count, modulus):
    """`count` device words uniform in [0, modulus)."""
    return torch.randint(0, modulus, (count,), generator=gen, device="cuda", dtype=torch.int64)


def _host(t):
    return t.cpu().numpy().view(np.uint64)


def _client_keys(gen, r, N1):
    N2, levels = N // 2 // N1, r.bit_length() - 1
    baby = torch.empty((N1 // 2, 6, 2 * N), device="cuda", dtype=torch.int64)
    baby[:, :3] = _words(gen, N1 // 2 * 3 * 2 * N, kb.CRTMOD).view(N1 // 2, 3, 2 * N)
    baby[:, 3:] = _words(gen, N1 // 2 * 3 * 2 * N, kb.BSMOD).view(N1 // 2, 3, 2 * N)
    return (_host(baby.view(-1)), _host(_words(gen, (N2 - 1) * 2 * 2 * N, kb.CRTMOD)),
            _host(_words(gen, levels * 4 * 2 * N, kb.CRTMOD)), _host(_words(gen, 4 * 2 * N, kb.CRTMOD)))


def _queries(gen, n):
    crt = _words(gen, n * 2 * N, kb.CRTMOD).view(n, 2 * N)
    bs = _words(gen, n * 2 * N, kb.BSMOD).view(n, 2 * N)
    return torch.cat([crt, bs], dim=1).contiguous()


def prepare(case, seed):
    kind, r, N1, n = case["kind"], case["r"], case["N1"], case["n"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    inflight = {"overlap": STREAMS, "batch": n, "hosted": n}.get(kind, 1)
    ctx = kb.Context(r, N1, max_clients=case["clients"], max_inflight=inflight)
    s = dict(case=case, ctx=ctx)
    if kind == "clients":
        # ternary secrets modulo crtMod, rows to fetch, responses to decrypt
        t = torch.randint(-1, 2, (n, N), generator=gen, device="cuda", dtype=torch.int64)
        s["secrets"] = _host(torch.where(t < 0, t + kb.CRTMOD, t))
        s["rows"] = torch.randint(0, N // 2, (n,), generator=gen, device="cuda").cpu().numpy().astype(np.uint32)
        s["responses"] = _host(_words(gen, n * 2 * N, kb.CRTMOD).view(n, 2 * N))
        s["seed"] = int(seed) & 0xFFFFFFFF
        return s
    raw = _words(gen, r * N * N // 2, 65537)
    torch.cuda.synchronize()
    ctx.preprocess_db_device(raw.data_ptr(), raw.numel())
    if kind == "refresh":
        s["raw"] = raw
    ctx.upload_perms(kb.permutation_matrix(N1))
    keys = [_client_keys(gen, r, N1) for _ in range(case["clients"])]
    s["cl"] = np.arange(n, dtype=np.int32) % case["clients"]
    queries = _queries(gen, n)
    for i, k in enumerate(keys):
        ctx.upload_client(i, *k)
    if kind in ("overlap", "batch"):
        s["queries"] = queries
        s["out"] = torch.empty((n, 2 * N), device="cuda", dtype=torch.int64)
        s["streams"] = [torch.cuda.Stream() for _ in range(STREAMS if kind == "overlap" else 1)]
    else:
        s["queries"] = _host(queries)
        s["out"] = np.empty((n, 2 * N), np.uint64)
    if case.get("tuned"):
        ctx.tune_batch(n)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass

def _signed(a):
    """The same words as int64 (all are below 2^63)."""
    return a.view(np.int64)


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind, r, n = case["kind"], case["r"], case["n"]
    if kind == "single":
        return _signed(ctx.answer(0, s["queries"][0], s["out"][0]))
    if kind == "overlap":
        for i in range(n):
            ctx.answer_device(int(s["cl"][i]), s["queries"][i].data_ptr(), s["out"][i].data_ptr(),
                              s["streams"][i % STREAMS].cuda_stream)
        return s["out"]
    if kind == "batch":
        ctx.answer_batch_device(s["cl"], s["queries"].data_ptr(), s["out"].data_ptr(), s["streams"][0].cuda_stream)
        return s["out"]
    if kind == "hosted":
        return _signed(ctx.answer_batch(s["cl"], s["queries"], s["out"]))
    if kind == "refresh":
        ctx.preprocess_db_device(s["raw"].data_ptr(), s["raw"].numel())
        return _signed(ctx.answer(0, s["queries"][0], s["out"][0]))
    if kind == "staged":
        first, switched = ctx.matrix_vector_mul(0, s["queries"][0])
        ext, coef = ctx.external_product(0, np.zeros(r * 2 * N, np.uint64), first)
        merged = np.empty(r * 2 * N, np.uint64)
        resp = ctx.packing(0, ext, merged)
        return dict(first=_signed(first), query=_signed(switched), ext=_signed(ext), coef=_signed(coef),
                    merged=_signed(merged), response=_signed(resp))
    made = ctx.client_queries(s["secrets"], s["rows"], s["seed"])
    messages = ctx.client_decrypt(s["secrets"], s["responses"], r)
    return dict(queries=_signed(made), messages=_signed(messages))


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _answer_ops(r, N1):
    """Integer operations of one answer: transforms (a butterfly is a product,
    a sum and a difference), key products and the database products."""
    N2, levels = N // 2 // N1, r.bit_length() - 1
    transforms = 15 + 11 + 6 * (N1 - 1) + 6 * r * (N2 - 1) + 12 * r + 14 * (r - 1)
    key_products = N * ((N1 - 1) * 3 * 2 * 3 + r * (N2 - 1) * 2 * 2 * 2 + r * 4 * 2 * 2 + (r - 1) * 4 * 2 * 2)
    return transforms * 3 * (N // 2) * 12 + 2 * key_products + 2 * 4 * r * N * N // 2 + levels


def work(case):
    kind, r, N1, n = case["kind"], case["r"], case["N1"], case["n"]
    N2, levels = N // 2 // N1, r.bit_length() - 1
    if kind == "clients":
        transforms = n * (3 + 3 + 5 + 4 * 2)
        return dict(bytes=n * 8 * N * (1 + 4 + 1 + 2 + 1), flops=transforms * 3 * (N // 2) * 12)
    db = r * N * N // 2 * 8
    key = 4 * N * (N1 // 2 * 3 * 2 * 3 + (N2 - 1) * 2 * 2 * 2 + levels * 4 * 2 * 2 + 4 * 2 * 2)
    passes = n if kind == "overlap" else 1      # answers of their own read the database each
    moved = passes * db + min(n, case["clients"]) * key + n * 8 * N * (4 + 2)
    ops = n * _answer_ops(r, N1)
    if kind == "refresh":
        moved += 2 * db                         # the raw words in, the preprocessed ones out
        ops += r * (N // 2) * 3 * 3 * (N // 2) * 12
    if kind == "staged":
        moved += 8 * N * r * 2 * 6              # the host buffers of the three calls
    return dict(bytes=moved, flops=ops)


def exact(case, seed):
    """None: every output is whole numbers, without rounding, so two builds are
    compared word for word."""
    return None
