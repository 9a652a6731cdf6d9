"""RZE decode at the edges of its chunk, bitmap and staging layout: byte counts
around every level's granularity, zero / sparse / dense / incompressible
(stored raw) contents, streams at 16-byte and 4-byte alignment, and streams
cut short (reported as malformed, never read past their end)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 7, 9, 64, 65, 511, 513, 4095, 4097, 16376, 16383, 16384, 16385, 32768 + 130, 5 * 16384 - 1]


def _data(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "zero":
        return np.zeros(n, np.uint8)
    if kind == "noise":
        return rng.integers(0, 256, n).astype(np.uint8)
    d = np.where(rng.random(n) < (0.02 if kind == "sparse" else 0.7), rng.integers(1, 256, n), 0).astype(np.uint8)
    d[-1] = 9  # the last byte of the last chunk counts
    return d


@pytest.mark.parametrize("kind", ["zero", "sparse", "dense", "noise"])
@pytest.mark.parametrize("n", SIZES)
def test_decode_edges(cuda, n, kind):
    from fzgpumodules_b200 import kernels as K
    d = _data(kind, n, n)
    stream = torch.from_numpy(np.ascontiguousarray(O.rze_encode(d))).to(cuda)
    assert np.array_equal(K.rze_decode(stream, n).cpu().numpy(), d)
    room = torch.zeros(stream.numel() + 4, dtype=torch.uint8, device=cuda)
    room[4:] = stream  # 4 bytes off the 16-byte boundary
    assert np.array_equal(K.rze_decode(room[4:], n).cpu().numpy(), d)


@pytest.mark.parametrize("kind", ["sparse", "noise"])
def test_decode_of_cut_stream_is_malformed(cuda, kind):
    from fzgpumodules_b200 import kernels as K
    n = 3 * 16384
    stream = np.ascontiguousarray(O.rze_encode(_data(kind, n, 5)))
    ws = K.Workspace()
    d = torch.from_numpy(stream).to(cuda)
    K.rze_decode(d, n, ws=ws)
    assert ws.status() == 0
    K.rze_decode(d[: stream.size - 40], n, ws=ws)
    assert ws.status() != 0
