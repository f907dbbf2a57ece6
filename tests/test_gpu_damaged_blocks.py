"""Damaged blocks of a byte stream, in every way the decoder takes blocks: a
block whose entry does not fit the stream or whose lane state was changed is
reported, every other block is decoded, and the next call is unaffected.

The damage is of the kinds that the decoder's own checks catch before or
after decoding: entries are compared with the header, and a changed state
ends in another position or state."""
import numpy as np
import pytest

import mans_b200 as mb
from tests.helpers import to_dev, to_host

pytestmark = pytest.mark.gpu

SMS = 148
BLOCK = 4096
CORRUPT = 10  # MANS_ERR_CORRUPT


def _bytes(n, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    u = torch.rand(n, device="cuda", generator=g)
    return torch.log1p(-u).div_(float(np.log1p(-0.05))).floor_().clamp_(0, 255).to(torch.uint8)


def _damage(s, kind, blocks):
    """A copy of stream s (device bytes) with the entries of `blocks` damaged."""
    import torch
    nb = int(to_host(s[:32]).view(np.uint32)[1])
    d = s.clone()
    for b in blocks:
        at = 32 + 512 + 128 * nb + 8 * b  # {bytes << 16 | words, first word}
        e = to_host(s[at:at + 8]).view(np.uint32).copy()
        if kind == "size":
            e[0] -= 1 << 16
        elif kind == "prefix":
            e[1] += 4
        if kind == "state":
            at = 32 + 512 + 128 * b + 4 * (b % 32)
            e = to_host(s[at:at + 4]).view(np.uint32).copy()
            e[0] ^= 1
        d[at:at + e.nbytes] = to_dev(e.view(np.uint8))
    torch.cuda.synchronize()
    return d


def _blocks(nb):
    """First and second of a pair, among the first and the claimed blocks, and the last ones."""
    return sorted({0, 3, nb // 2 & ~1, (nb * 3 // 4) | 1, nb - 2, nb - 1} & set(range(nb)))


def _check(out, x, bad):
    """out equals x but for the blocks `bad`, of which one is wrong at least."""
    import torch
    wrong = torch.nonzero(out != x).flatten().div(BLOCK, rounding_mode="floor").unique().tolist()
    assert set(wrong) <= set(bad), (wrong[:8], bad)


# blocks: the words staged whole, a block per warp, pairs of blocks with claims
@pytest.mark.parametrize("p", [9, 10, 11])
@pytest.mark.parametrize("blocks", [3, 7, SMS * 12, SMS * 24, SMS * 31 + 5, SMS * 40, SMS * 130 + 1])
@pytest.mark.parametrize("kind", ["size", "prefix", "state"])
def test_damaged_block_costs_no_other(kind, blocks, p):
    import torch
    n = blocks * BLOCK - 1000
    x = _bytes(n, blocks)
    w = mb.Workspace(n)
    try:
        s = mb.compress(x, p, ws=w)
        bad = _blocks(blocks)
        d = _damage(s, kind, bad)
        out = torch.full((n,), 238, dtype=torch.uint8, device="cuda")
        mb.decompress_into(w, d, d.numel(), out)
        st, detail = w.status()
        assert st == CORRUPT and detail in bad
        _check(out, x, bad)
        out.fill_(0)
        mb.ansDecode(p, d, out)
        st, detail = mb.ans_last_status()
        assert st == CORRUPT and detail in bad
        _check(out, x, bad)
        mb.decompress_into(w, s, s.numel(), out)
        assert w.status()[0] == 0 and torch.equal(out, x)
    finally:
        w.close()


# big: bytes of a buffer that sets the chunk size (8 blocks, 32, pairs of 64 and 128)
@pytest.mark.parametrize("kind", ["size", "prefix", "state"])
@pytest.mark.parametrize("big", [0, 24_000_000, 80_000_000, 320_000_000])
def test_batch_damaged_block_costs_no_other(kind, big):
    import torch

    from mans_b200.batch import Batch
    sizes = [BLOCK * 5 - 1, BLOCK * 70, BLOCK * 200 + 17, 1] + ([big] if big else [])
    xs = [_bytes(n, n) for n in sizes]
    ss = [mb.compress(x, 9 + i % 3) for i, x in enumerate(xs)]
    bad = {i: _blocks(-(-n // BLOCK)) for i, n in enumerate(sizes) if i in (1, 2, 4)}
    ds = [_damage(s, kind, bad[i]) if i in bad else s for i, s in enumerate(ss)]
    b = Batch(len(xs), sum(sizes))
    try:
        for streams, damaged in ((ds, bad), (ss, {})):
            outs = [torch.full((n,), 238, dtype=torch.uint8, device="cuda") for n in sizes]
            b.decompress_async(Batch.decompress_items(streams, [s.numel() for s in streams], outs))
            _, st, detail = b.status(len(xs))
            for i, (x, out) in enumerate(zip(xs, outs)):
                if i in damaged:
                    assert st[i] == CORRUPT and detail[i] in damaged[i]
                    _check(out, x, damaged[i])
                else:
                    assert st[i] == 0 and torch.equal(out, x)
    finally:
        b.close()
