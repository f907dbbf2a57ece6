"""The byte coder's kernels at the sizes where their work split changes: the
warps per CTA (up to 32 a multiprocessor), the decoder's pairs of blocks and
the word pieces of 256 words, and the batch decoder's chunk sizes, against the
oracle, byte for byte."""
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


@pytest.mark.parametrize("p", [9, 10, 11])
@pytest.mark.parametrize("tail", [-4096 * 3 - 511, -1, 0, 1, 512, 4096])
def test_decoder_pairs(ws, oracle, tail, p):
    """Around two waves of pairs, through both decode calls; the last blocks
    (one of an odd number, a partial one) are decoded singly."""
    import torch
    n = 2 * 64 * SMS * 4096 // 3 + tail
    x = W.random_bytes(n, 7 + p, ("sparse", "two", "skewed")[p - 9])
    ref = oracle.ans_encode(x, p)
    s = to_dev(ref)
    np.testing.assert_array_equal(to_host(mb.decompress(s, n, torch.uint8, ws=ws)), x)
    out = torch.zeros(n, dtype=torch.uint8, device="cuda")
    mb.ansDecode(p, s, out)
    assert mb.ans_last_status()[0] == 0
    np.testing.assert_array_equal(to_host(out), x)


@pytest.mark.parametrize("n", [1 << 20, 1_000_003])
def test_single_symbol_keeps_its_state(ws, oracle, n):
    """A pdf of 2^p (one symbol) is the slot table's special entry."""
    import torch
    x = np.full(n, 200, np.uint8)
    s = mb.compress(to_dev(x), 11, ws=ws)
    np.testing.assert_array_equal(to_host(s), oracle.ans_encode(x, 11))
    np.testing.assert_array_equal(to_host(mb.decompress(s, n, torch.uint8, ws=ws)), x)


@pytest.mark.parametrize("big", [0, 900_000, 6_000_000, 24_000_000, 400_000_000])
def test_batch_decoder_chunks(oracle, big):
    """Chunks of 8 to 128 blocks: a few small buffers of every type and
    precision beside one of `big` bytes that sets the chunk size."""
    import torch

    from mans_b200.batch import Batch
    xs, ps = [], []
    for i, n in enumerate([1, 4095, 4096 * 8 + 1, 4096 * 33, 4096 * 66 - 5, 70_001, 600_000]):
        xs += [W.random_bytes(n, i, "skewed"), W.gradient_u16(n, i), W.quant_u32(n // 2 + 1, i)]
        ps += [9 + i % 3] * 3
    refs = [to_dev(oracle.ans_encode(x, p) if x.dtype == np.uint8 else oracle.compress(x, p))
            for x, p in zip(xs, ps)]
    tdt = {np.uint8: torch.uint8, np.uint16: torch.uint16, np.uint32: torch.uint32}
    dt = [tdt[x.dtype.type] for x in xs]
    big_in = None
    if big:  # made on the device, compressed by the library itself
        g = torch.Generator(device="cuda")
        g.manual_seed(big)
        big_in = torch.randint(0, 50, (big,), dtype=torch.uint8, device="cuda", generator=g)
        refs.append(mb.compress(big_in, 10))
        dt.append(torch.uint8)
    sizes = [x.size for x in xs] + ([big] if big else [])
    b = Batch(32, sum(x.nbytes for x in xs) + big)
    try:
        outs = b.decompress(refs, list(zip(sizes, dt)))
        for x, y in zip(xs, outs):
            np.testing.assert_array_equal(to_host(y, x.dtype), x)
        assert big_in is None or torch.equal(outs[-1], big_in)
    finally:
        b.close()


@pytest.mark.parametrize("n", [512, 511, 512 * 37, 512 * 37 + 300])
@pytest.mark.parametrize("spread", [0, 126, 127, 300])
def test_u32_groups_of_one_byte_codes(ws, oracle, n, spread):
    """Groups at and around the limit of one code byte per element, high and
    low centers, mixed with groups that need more."""
    import torch
    rng = np.random.default_rng(n + spread)
    x = np.empty(n, np.uint32)
    for g in range(0, n, 512):
        m = min(512, n - g)
        c = int(rng.choice([0, 130, 70_000, (1 << 32) - 1 - 2 * spread]))
        v = c + spread + rng.integers(-spread, spread + 1, m) * (rng.random(m) < 0.05)
        x[g:g + m] = np.clip(v, 0, (1 << 32) - 1).astype(np.uint32)
    s = mb.compress(to_dev(x), 10, ws=ws)
    np.testing.assert_array_equal(to_host(s), oracle.compress(x, 10))
    np.testing.assert_array_equal(to_host(mb.decompress(s, n, torch.uint32, ws=ws), np.uint32), x)


@pytest.mark.parametrize("byte", [0, 254, 255])
def test_u32_one_byte_group_with_a_bad_code(ws, byte):
    """A byte that is no code in a group of 16-byte records is reported."""
    import torch
    x = np.full(1024, 1000, np.uint32)
    m = to_host(mb.adm_map(to_dev(x), ws=ws)).copy()
    assert m.size == 80 + 1024
    for at in (80, 80 + 511, 80 + 700):
        bad = m.copy()
        bad[at] = byte
        with pytest.raises(mb.MansError) as e:
            mb.adm_unmap(to_dev(bad), x.size, torch.uint32, ws=ws)
        assert e.value.code == 10  # MANS_ERR_CORRUPT
    np.testing.assert_array_equal(to_host(mb.adm_unmap(to_dev(m), x.size, torch.uint32, ws=ws), np.uint32), x)


@pytest.mark.parametrize("kind", ["detector", "quant", "near", "wide"])
@pytest.mark.parametrize("n", [(1 << 21) - 1, 1 << 21, 4608 * 512, 4608 * 512 + 1, (1 << 22) + 777])
def test_u32_records_gathered_by_the_encoder(oracle, n, kind):
    """The two ways a uint32 compress can go, at their border and where the
    records begin on a block's start (4,608 groups); a workspace without room
    for the slots takes the other way, to the same bytes."""
    import torch
    rng = np.random.default_rng(n)
    x = {"detector": lambda: W.detector_u32(n, 1), "quant": lambda: W.quant_u32(n, 2),
         "near": lambda: rng.integers(0, 90, n).astype(np.uint32),
         "wide": lambda: rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)}[kind]()
    ref = oracle.compress(x, 10)
    d = to_dev(x)
    groups = -(-n // 512)
    for merged in (0, 4000 * groups if kind != "wide" else 0):
        w = mb.Workspace(4 * n, merged)
        try:
            s = mb.compress(d, 10, ws=w)
            np.testing.assert_array_equal(to_host(s), ref)
            y = mb.decompress(s, n, torch.uint32, ws=w)
        finally:
            w.close()
        np.testing.assert_array_equal(to_host(y, np.uint32), x)


@pytest.mark.parametrize("b", [40, 160, 280, 420, 800])
@pytest.mark.parametrize("layout", [0, 1, 2])
def test_u16_streams_around_their_word_limits(ws, oracle, b, layout):
    """Lane streams whose halves stay below, pass 32 bits and whose sum passes
    64; ragged end."""
    import torch
    n = 100_003
    rng = np.random.default_rng(b)
    scale = np.repeat(rng.choice([0.05, 1.0], -(-n // 8)), 8)[:n]  # per eight elements
    x = np.clip(np.round(30000 + rng.laplace(0, 1, n) * b * scale), 0, 65535).astype(np.uint16)
    s = mb.compress(to_dev(x), 10, ws=ws, layout=layout)
    np.testing.assert_array_equal(to_host(s), oracle.compress(x, 10, layout))
    y = mb.decompress(s, n, torch.uint16, ws=ws, layout=layout)
    np.testing.assert_array_equal(to_host(y, np.uint16), x)


@pytest.mark.parametrize("p", [9, 10, 11])
@pytest.mark.parametrize("blocks", [1, 8, 9, 24 * SMS - 1, 24 * SMS, 24 * SMS + 1, 64 * SMS + 1])
@pytest.mark.parametrize("tail", [0, -4090])
def test_decoder_kernels(ws, oracle, blocks, tail, p):
    """The decoder's two kernels (three CTAs of eight warps per multiprocessor,
    or one of 32) at the sizes where one takes over from the other, full and
    short last blocks."""
    import torch
    n = blocks * 4096 + tail
    x = W.random_bytes(n, blocks + p, ("uniform", "sparse", "skewed")[p - 9])
    s = to_dev(oracle.ans_encode(x, p))
    for _ in range(2):  # the second call finds the work counters reset
        np.testing.assert_array_equal(to_host(mb.decompress(s, n, torch.uint8, ws=ws)), x)


@pytest.mark.parametrize("p", [9, 10, 11])
@pytest.mark.parametrize("kind,n", [("wide", 3_400_000), ("wide", 4_700_001), ("near", 5_500_003)])
def test_decoder_block_count_off_the_estimate(kind, n, p):
    """Many more blocks than estimated from the value count (a warp of the small
    kernel takes several), and many fewer (the large one's warps one at most).
    The stream is the library's own; a damaged one is refused between."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    hi = 90 if kind == "near" else 2**31 - 1
    x = torch.randint(0 if kind == "near" else -2**31, hi, (n,), dtype=torch.int32, device="cuda",
                      generator=g).view(torch.uint32)
    w = mb.Workspace(4 * n)
    try:
        s = mb.compress(x, p, ws=w)
        nb = int(to_host(s[:32]).view(np.uint32)[1])
        est = -(-3 * n // 4096)
        if kind == "near":
            assert nb < 15 * SMS and est > 24 * SMS
        else:
            assert nb > 24 * SMS and est <= 24 * SMS
        bad = s.clone()
        for b in (0, nb // 2, nb - 1):
            bad[32 + 512 + 128 * nb + 8 * b + 2] ^= 1  # the block's byte count
        y = torch.empty_like(x)
        mb.decompress_into(w, bad, bad.numel(), y)
        assert w.status()[0] == 10  # MANS_ERR_CORRUPT
        assert torch.equal(mb.decompress(s, n, torch.uint32, ws=w), x)
    finally:
        w.close()


@pytest.mark.parametrize("kind", ["wide", "near", "quant"])
@pytest.mark.parametrize("n", [150_000, 1_000_001, (1 << 21) - 1, 3 << 20])
def test_encoder_block_count_off_the_estimate(oracle, n, kind):
    """uint32 data of one to five mapped bytes a value, for which the encoder's
    CTAs are launched alike: with blocks for some of their warps, all, or several
    rounds, on both sides of the size from which it gathers the records."""
    import torch
    rng = np.random.default_rng(n)
    x = {"wide": lambda: rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32),
         "near": lambda: rng.integers(0, 90, n).astype(np.uint32),
         "quant": lambda: W.quant_u32(n, 5)}[kind]()
    w = mb.Workspace(4 * n)
    try:
        for p in (9, 11):
            s = mb.compress(to_dev(x), p, ws=w)
            np.testing.assert_array_equal(to_host(s), oracle.compress(x, p))
    finally:
        w.close()


def _groups_at_the_limits(n, seed):
    """uint32 groups whose values reach exactly to 125, 126, 127 or 300 from their
    center on either side, at low, middle and the highest centers; a few values of
    every group sit at the limits, as many below as above, and the rest at the
    center, so that the truncated mean is the center."""
    rng = np.random.default_rng(seed)
    x = np.empty(n, np.uint32)
    for g in range(0, n, 512):
        m = min(512, n - g)
        d = int(rng.choice([0, 1, 125, 126, 127, 300]))
        c = int(rng.choice([d, 130 + d, 70_000, 1 << 31, (1 << 32) - 1 - d]))
        v = np.full(m, c, np.int64)
        k = int(rng.integers(0, min(m // 2, 9)))
        at = rng.permutation(m)
        v[at[:k]] = c - d
        v[at[k:2 * k]] = c + d
        x[g:g + m] = v
    return x


@pytest.mark.parametrize("p", [9, 10, 11])
@pytest.mark.parametrize("n", [(1 << 21) - 512, 1 << 21, (1 << 21) + 300])
def test_u32_split_groups_at_the_limits(oracle, n, p):
    """The short path of the uint32 map that leaves records in slots, at its
    limits, and the gathering encoder at every precision."""
    import torch
    x = _groups_at_the_limits(n, n + p)
    assert int(x.min()) == 0 and int(x.max()) == (1 << 32) - 1
    codes = oracle.adm_u32_map(x[:1 << 20])
    assert (codes == 253).any() and (codes == 252).any()  # 126 below and above
    w = mb.Workspace(4 * n)
    try:
        s = mb.compress(to_dev(x), p, ws=w)
        np.testing.assert_array_equal(to_host(s), oracle.compress(x, p))
        y = mb.decompress(s, n, torch.uint32, ws=w)
    finally:
        w.close()
    np.testing.assert_array_equal(to_host(y, np.uint32), x)
