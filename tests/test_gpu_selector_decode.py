"""Decoding selector containers: chunk and block sizes around every coder's
granularity, and containers with a fault, which are refused."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 767, 769, 8191, 8193, 16384, 32767, 32768, 32769, 3 * 32768 + 20001]


def Sel():
    from fzgpumodules_b200 import selector
    return selector


def _codes(kind, n):
    rng = np.random.default_rng(n)
    if kind == 0:  # Bitshuffle + RZE: sparse
        return np.where(rng.random(n) < 0.02, rng.integers(0, 60000, n), 0).astype(np.uint16)
    if kind == 1:  # RLE: runs of 1 .. 400
        return np.repeat(rng.integers(0, 900, n), rng.integers(1, 400, n))[:n].astype(np.uint16)
    if kind == 2:  # Bitpack: 2 bits
        return rng.integers(0, 4, n).astype(np.uint16)
    return np.minimum(rng.geometric(0.3, n), 1023).astype(np.uint16)  # Huffman


@pytest.mark.parametrize("kind", range(4))
@pytest.mark.parametrize("n", SIZES)
def test_roundtrip_edges(cuda, n, kind):
    c = _codes(kind, n)
    d = torch.from_numpy(c).to(cuda)
    for mode in (Sel().fixed(kind), Sel().EXHAUSTIVE):
        blob, _ = Sel().encode(d, mode)
        assert np.array_equal(Sel().decode(blob, n).cpu().numpy(), c)


@pytest.mark.parametrize("kind", range(4))
def test_faults_are_refused(cuda, kind):
    from fzgpumodules_b200._lib import FzbError
    n = 3 * 32768
    blob, tags = Sel().encode(torch.from_numpy(_codes(kind, n)).to(cuda), Sel().fixed(kind))
    assert set(tags.cpu().tolist()) == {kind}
    pad = 4  # tags and params of three chunks
    first = 16 + 2 * pad + 4 * 3  # the first payload

    def bad(change):
        b = blob.clone()
        b = change(b)
        with pytest.raises(FzbError):
            Sel().decode(b, n)

    def put(at, v):
        def f(b):
            b[at] = v
            return b
        return f
    bad(put(0, 0))                      # magic
    bad(put(16 + 1, 9))                 # tag
    bad(lambda b: b[: b.numel() - 8])   # cut short
    if kind == 2:
        bad(put(16 + pad + 1, 5))       # bits a code (a Bitpack payload has no header)
    else:
        bad(put(first, 77))             # the first payload's own header


@pytest.mark.parametrize("kind", range(4))
def test_chunk_with_a_gap_behind_its_payload(cuda, kind):
    """A chunk's size in the container may be any that fits the container (here
    over 4 MiB): the next payload starts behind it."""
    n = 3 * 32768
    c = _codes(kind, n)
    blob, _ = Sel().encode(torch.from_numpy(c).to(cuda), Sel().fixed(kind))
    b = blob.cpu().numpy()
    at = 16 + 2 * 4  # three sizes behind the tags and params
    sizes = b[at: at + 12].view(np.uint32).copy()
    cut = at + 12 + (int(sizes[0]) + 3) // 4 * 4
    gap = np.zeros(5 << 20, np.uint8)
    wide = np.concatenate([b[:cut], gap, b[cut:]])
    wide[at: at + 4] = np.array([cut - at - 12 + gap.size], np.uint32).view(np.uint8)
    got = Sel().decode(torch.from_numpy(wide).to(cuda), n).cpu().numpy()
    assert np.array_equal(got, c)
