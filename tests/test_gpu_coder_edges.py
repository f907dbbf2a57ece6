"""The byte coder's kernels at the sizes where their work split changes: the
encoder's warps per CTA (4 to 32 a multiprocessor) and its word pieces of 256
words, against the oracle, byte for byte."""
import numpy as np
import pytest

import mans_b200 as mb
from mans_b200 import workloads as W
from tests.helpers import to_dev, to_host

pytestmark = pytest.mark.gpu

SMS = 148


@pytest.fixture(scope="module")
def ws():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    w = mb.Workspace(64 << 20)
    yield w
    w.close()


def _words_per_block(n, p):
    """Bytes whose blocks code to more and more words: symbol 0 has nearly all
    of the probability, every other symbol costs p bits."""
    x = np.zeros(n, np.uint8)
    for b in range(-(-n // 4096)):
        k = min(4096, n - b * 4096)
        rare = min(k, 16 * b)  # p * rare / 16 words
        x[b * 4096:b * 4096 + rare] = 1 + np.arange(rare) % 255
    return x


@pytest.mark.parametrize("p", [9, 10, 11])
@pytest.mark.parametrize("blocks,tail", [(1, -1), (4 * SMS, 0), (4 * SMS, 1), (9 * SMS, 37),
                                         (32 * SMS, -4095), (32 * SMS + 1, 33)])
def test_encoder_split(ws, oracle, blocks, tail, p):
    import torch
    n = blocks * 4096 + tail
    kind = ("skewed", "uniform", "sparse")[p - 9]
    x = W.random_bytes(n, blocks + p, kind)
    s = mb.compress(to_dev(x), p, ws=ws)
    np.testing.assert_array_equal(to_host(s), oracle.ans_encode(x, p))
    np.testing.assert_array_equal(to_host(mb.decompress(s, n, torch.uint8, ws=ws)), x)


@pytest.mark.parametrize("p", [9, 10, 11])
def test_encoder_word_pieces(ws, oracle, p):
    import torch
    n = 257 * 4096 - 5
    x = _words_per_block(n, p)
    ref, bw = oracle.ans_encode(x, p, with_block_words=True)
    assert int(bw.min()) < 256 and int(bw.max()) > 2048
    s = mb.compress(to_dev(x), p, ws=ws)
    np.testing.assert_array_equal(to_host(s), ref)
    np.testing.assert_array_equal(to_host(mb.decompress(s, n, torch.uint8, ws=ws)), x)
