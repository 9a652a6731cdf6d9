"""Huffman encoders at the edge of joining four codes into one word (32 bits in
all): partitions where every four just fit, where one four does not, and where all
of a warp's are long, against the oracle's bytes."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

LEAVES = 26


def _book():
    f = np.zeros(1024, np.uint32)
    a, b = 1, 1
    for i in range(LEAVES):  # code lengths 25, 25, 24, ..., 1
        f[i] = a
        a, b = b, a + b
    bk4, rb = O.huff_book(f, 1024)
    return bk4, rb, (bk4 >> 27).astype(int)


@pytest.mark.parametrize("fine", [False, True])
@pytest.mark.parametrize("kind", ["fit", "one over", "over", "mixed", "short"])
def test_four_codes_at_a_word(cuda, kind, fine):
    from fzgpumodules_b200 import kernels as K
    bk4, rb, length = _book()
    sym = {int(l): i for i, l in enumerate(length[:LEAVES])}  # a symbol of each length
    assert sorted(sym) == list(range(1, LEAVES))
    fit = [(8, 8, 8, 8), (16, 14, 1, 1), (1, 1, 14, 16), (20, 10, 1, 1), (1, 25, 5, 1), (2, 2, 14, 14), (1, 1, 15, 15),
           (25, 5, 1, 1), (1, 2, 4, 25)]  # 32 bits each
    over = [(8, 8, 8, 9), (9, 8, 8, 8), (1, 1, 16, 15), (25, 25, 25, 25), (16, 15, 1, 1)]
    assert all(sum(q) == 32 for q in fit) and all(sum(q) > 32 for q in over)
    rng = np.random.default_rng(len(kind))
    n4 = 768 * 40
    pick = lambda qs: [qs[i] for i in rng.integers(0, len(qs), n4)]  # noqa: E731
    quads = pick(over if kind == "over" else fit)
    if kind == "one over":
        for i in rng.choice(n4, 25, replace=False):
            quads[i] = over[i % len(over)]
    if kind == "mixed":
        quads = [over[i % 5] if rng.random() < 0.4 else q for i, q in enumerate(quads)]
    if kind == "short":
        quads = [(1, 1, 1, 1) if i % 3 else (2, 1, 3, 1) for i in range(n4)]
    codes = np.array([sym[l] for q in quads for l in q], np.uint16)
    for n in (codes.size, codes.size - 1, 768 * 3 + 2, 1024 * 3 + 3):
        ref = O.huff_encode(codes[:n], 1024, bk4, rb, 1024 if fine else 768)
        d = torch.from_numpy(codes[:n].copy()).to(cuda)
        blob, _ = K.huff_encode(d, bk4, rb, 1024, fine=fine)
        assert np.array_equal(blob.cpu().numpy(), ref)
        assert np.array_equal(K.huff_decode(blob, n, 1024).cpu().numpy(), codes[:n])


@pytest.mark.parametrize("symbols", [255, 256, 257, 300, 512, 1024])
def test_selector_packing_at_a_word(cuda, symbols):
    """Equally frequent symbols: codes of 8 bits for 256, the longest that join."""
    from fzgpumodules_b200 import selector as S
    n = 32768 + 5000
    rng = np.random.default_rng(symbols)
    c = np.concatenate([rng.permutation(np.arange(n) % symbols)]).astype(np.uint16)
    blob, tags = S.encode(torch.from_numpy(c).to(cuda), S.fixed(3))
    b, t = blob.cpu().numpy(), tags.cpu().numpy()
    sizes = b[16 + 8: 16 + 16].view(np.uint32)
    off = 16 + 8 + 8
    for i in range(2):
        chunk = c[32768 * i: 32768 * (i + 1)]
        if t[i] == 3:  # (where it fits)
            f, _ = O.histogram(chunk, 1024)
            ref = O.huff_encode(chunk, 1024, *O.huff_book(f, 1024))
            assert np.array_equal(b[off: off + ref.size], ref)
        off += (int(sizes[i]) + 3) & ~3
    assert t[0] == 3
    assert np.array_equal(S.decode(blob, n).cpu().numpy(), c)
