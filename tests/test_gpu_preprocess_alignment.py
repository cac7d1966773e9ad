"""Database preprocessing from device pointers that are 16-byte aligned and
8-byte aligned only (the kernels read pairs of words where they can): the same
datacrt, equal to the oracle's; and invalid words found at the edges of the
validation pass's chunks in both."""
import numpy as np
import pytest

import kspir_b200 as kb
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
N = po.N
WORDS = N * N // 2


@pytest.mark.parametrize("N1", [64, 128, 256])
@pytest.mark.parametrize("offset", [0, 1])
def test_datacrt_from_any_word_alignment(N1, offset):
    rng = np.random.default_rng(400 + N1)
    raw = rng.integers(0, 65537, WORDS, dtype=np.uint64)
    raw[:9] = [0, 1, 32767, 32768, 32769, 65535, 65536, 65536, 0]
    want = po.db_preprocess(raw, 1, N1)
    d = torch.empty(WORDS + 2, dtype=torch.int64, device="cuda")
    d[offset:offset + WORDS] = torch.from_numpy(raw.view(np.int64)).cuda()
    torch.cuda.synchronize()
    with kb.Context(1, N1, max_inflight=2) as ctx:
        ctx.preprocess_db_device(d.data_ptr() + 8 * offset, WORDS)
        assert (ctx.download_db() == np.asarray(want).reshape(-1)).all()


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("where", [0, 1, WORDS // 2 + 1, WORDS - 2, WORDS - 1])
@pytest.mark.parametrize("value", [65537, 1 << 32, 1 << 63])
def test_invalid_words_are_found(offset, where, value):
    d = torch.zeros(WORDS + 2, dtype=torch.int64, device="cuda")
    d[offset + where] = value if value < 1 << 63 else -(1 << 63)
    torch.cuda.synchronize()
    with kb.Context(1, 128) as ctx:
        with pytest.raises(kb.KspirError):
            ctx.preprocess_db_device(d.data_ptr() + 8 * offset, WORDS)
        d[offset + where] = 65536
        torch.cuda.synchronize()
        ctx.preprocess_db_device(d.data_ptr() + 8 * offset, WORDS)
