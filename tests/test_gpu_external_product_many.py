"""The staged external product on both sides of the line between its kernels (one
ciphertext per CTA from more ciphertexts than SMs on, a CTA per prime below): nonzero
accumulators, both outputs, with zero, largest and random words.  Word for word against
the oracle for some ciphertexts of each call."""
import numpy as np
import pytest
import torch

import kspir_b200 as kb
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
N, R = po.N, 256


def test_counts_around_the_number_of_sms():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    keys = po.gen_client(801, R, 256)
    rng = np.random.default_rng(802)
    acc = rng.integers(0, po.CRTMOD, size=(R, 2 * N), dtype=np.uint64)
    first = rng.integers(0, po.CRTMOD, size=(R, 2 * N), dtype=np.uint64)
    first[0] = 0
    first[1], acc[1] = po.CRTMOD - 1, po.CRTMOD - 1
    acc[2] = 0
    with kb.Context(R, 256, max_clients=1, max_inflight=1) as ctx:
        ctx.upload_client(0, keys["baby"], keys["giant"], keys["packing"], keys["rgsw"])
        for count in (sms, sms + 1, R):
            ext, coef = (x.reshape(count, 2 * N) for x in ctx.external_product(0, acc[:count], first[:count]))
            for i in (0, 1, 2, count - 1):
                want, want_coef = po.external_product(first[i], keys["rgsw"], ext=acc[i])
                assert np.array_equal(ext[i], want), (count, i)
                assert np.array_equal(coef[i], want_coef), (count, i)
