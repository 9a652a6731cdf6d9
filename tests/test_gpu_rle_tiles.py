"""RLE at the edges of its tiles (4096 elements encoded, 1024 runs decoded)
against the oracle, exact bytes: sizes around a tile, a run that ends at, before
and after its edge, runs over whole tiles, one run and no runs shorter than two."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TDT = {np.uint8: torch.uint8, np.uint16: torch.uint16, np.uint32: torch.int32}


def _runs(lengths, dtype):
    v = (np.arange(len(lengths)) % 7 + 1).astype(dtype)
    return np.repeat(v, lengths)


def _cases(dtype):
    rng = np.random.default_rng(5)
    for n in (1, 2, 4095, 4096, 4097, 8191, 3 * 4096 + 1):
        yield _runs([n], dtype)                                   # one run
        yield (np.arange(n) % 5).astype(dtype)                    # no run of two
        yield np.repeat(rng.integers(0, 9, n).astype(dtype), 2)[:n]
    for d in (-1, 0, 1):
        yield _runs([4096 + d, 4096, 1, 4096 * 5 + d, 63, 64, 65, 2], dtype)
        yield _runs([1] * (1024 + d), dtype)                      # decoder tiles
        yield _runs([1] * (2047 + d) + [5000], dtype)
        yield _runs([3] * 1023 + [70000 + d] + [1, 2] * 700, dtype)


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.uint32])
def test_rle_tile_edges(cuda, dtype):
    from fzgpumodules_b200 import kernels as K
    for a in _cases(dtype):
        t = torch.from_numpy(a.view(np.int32) if dtype == np.uint32 else a).to(cuda)
        ref = O.rle_encode(a)
        enc, _ = K.rle_encode(t)
        assert np.array_equal(enc.cpu().numpy(), ref)
        dec = K.rle_decode(enc, a.size, TDT[dtype])
        assert np.array_equal(dec.cpu().numpy().view(dtype), a)


@pytest.mark.parametrize("n", [1024 * 1024 - 1, 4 * 1024 * 1024 + 1, 9 * 1024 * 1024 + 5])
def test_many_tiles_of_runs(cuda, n):
    """A thread's share of the sums' scan: one to twelve sums, the last share partial."""
    from fzgpumodules_b200 import kernels as K
    t = (torch.arange(n, device=cuda) % 251).to(torch.uint8)
    enc, _ = K.rle_encode(t)
    assert enc.numel() == 4 + (n + 3) // 4 * 4 + 4 * n
    assert torch.equal(K.rle_decode(enc, n, torch.uint8), t)
    t[n // 3: n // 3 + 5000] = 9
    enc, _ = K.rle_encode(t)
    assert torch.equal(K.rle_decode(enc, n, torch.uint8), t)


def test_long_runs_take_no_scan_of_all_tiles(cuda):
    """One run over the whole stream: 2^25 bytes cost little more than 2^24 16-bit codes."""
    from fzgpumodules_b200 import kernels as K

    def least(n, dtype):
        enc, _ = K.rle_encode(torch.zeros(n, dtype=dtype, device=cuda))
        times = []
        for _ in range(12):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(5):
                K.rle_decode(enc, n, dtype)
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times)
    t = least(1 << 24, torch.uint16), least(1 << 25, torch.uint8)
    print("us a call", [200 * v for v in t])
    assert t[1] < 1.85 * t[0]  # 1.6; 2.1 with a scan of all tiles
