"""Codes by tiles (fields of any rank and extents) against the oracle: extents
around the tile, load and chunk sizes, input at 16- and 4-byte alignment, few
and many outliers, NaN and infinities; the codes call and the fused chain, and
an input counted as padded without a padded copy."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

DIMS = [(31, 33, 1), (32, 64, 1), (36, 5, 1), (333, 130, 1), (8, 2000, 1), (9000, 3, 1),
        (3, 1, 1), (1023, 1, 1), (8192, 1, 1), (8193, 1, 1), (40961, 1, 1),
        (7, 9, 3), (8, 8, 8), (33, 17, 9), (64, 10, 21), (130, 5, 40), (100, 100, 9), (1, 5, 300)]


def _field(dims, seed, special):
    rng = np.random.default_rng(seed)
    n = int(np.prod(dims))
    x = np.cumsum(rng.normal(0, 0.02, n)).astype(np.float32)
    x[rng.integers(0, n, max(1, n // 100))] = 37.0
    if special:
        x[rng.integers(0, n, 3)] = [np.nan, np.inf, -np.inf]
    return x


def _same(got, ref):
    """Equal bits, but for a NaN's payload, which IEEE 754 leaves to the machine."""
    nan = np.isnan(ref)
    return np.array_equal(np.isnan(got), nan) and np.array_equal(got.view(np.uint32)[~nan], ref.view(np.uint32)[~nan])


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("radius", [32768, 40])
@pytest.mark.parametrize("dims", DIMS)
def test_codes_and_chain(cuda, dims, radius, special):
    from fzgpumodules_b200 import kernels as K
    x = _field(dims, 3 * int(np.prod(dims)) + radius, special)
    _, r, _ = O.resolve_eb(1e-2, O.ABS, 0.0)
    for zigzag, shift in ((True, 0), (False, 0), (True, 1)):
        codes, err, idx, cnt = O.lq_fwd(x, dims, r, radius, zigzag)
        room = torch.zeros(x.size + shift, device=cuda)
        room[shift:] = torch.from_numpy(x).to(cuda)
        for fused in (False, True):
            f = K.lq_bs_rze_compress if fused else K.lq_forward
            out = f(room[shift:], dims, 1e-2, K.ABS, radius, zigzag, 1.0)
            assert int(out["count"].item()) == cnt
            assert np.array_equal(out["idx"][:cnt].cpu().numpy().view(np.uint32), idx)
            assert _same(out["err"][:cnt].cpu().numpy(), err)
            if fused:
                stream = O.rze_encode(O.bitshuffle(codes, 16384, 2))
                assert np.array_equal(out["rze"][: int(out["rze_size"].item())].cpu().numpy(), stream)
            else:
                assert np.array_equal(out["codes"].cpu().numpy(), codes)


# fields that fill little of their tiles, on both sides of the line, rows a multiple
# of four elements and not, runs of 1024 elements ending inside the field
NARROW = [(1, 2, 1), (1, 5000, 1), (2, 3001, 1), (3, 1025, 1), (4, 2049, 1), (5, 999, 1), (7, 700, 1), (8, 601, 1),
          (16, 200, 1), (18, 130, 1), (19, 64, 1), (4100, 2, 1), (4099, 3, 1), (2000, 18, 1), (333, 19, 1),
          (1, 1, 5000), (1, 300, 9), (2, 2, 999), (3, 300, 7), (4, 4, 100), (4, 6, 90), (100, 2, 31), (1001, 1, 17),
          (1000, 3, 9), (33, 3, 40), (64, 64, 2), (65, 31, 3)]


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("radius", [32768, 40])
@pytest.mark.parametrize("dims", NARROW)
def test_narrow_fields(cuda, dims, radius, special):
    test_codes_and_chain(cuda, dims, radius, special)


def test_narrow_fields_in_a_batch(cuda):
    from fzgpumodules_b200 import kernels as K
    fields = [dict(x=torch.from_numpy(_field(d, 7 + i, False)).to(cuda), dims=d, eb=1e-2, mode=K.ABS,
                   radius=40 if i % 2 else 32768, zigzag=True)
              for i, d in enumerate(NARROW + [(100, 90, 1), (5000, 1, 1), (100, 41, 9)])]
    b = K.Batch(fields)
    b.launch()
    torch.cuda.synchronize()
    for f, o in zip(fields, b.outputs):
        r = K.lq_bs_rze_compress(f["x"], f["dims"], f["eb"], f["mode"], f["radius"], True, 0.2)
        size, cnt = int(r["rze_size"].item()), int(r["count"].item())
        assert int(o["rze_size"].item()) == size and torch.equal(o["rze"][:size], r["rze"][:size])
        assert int(o["count"].item()) == cnt
        kept = min(cnt, r["cap"])
        assert torch.equal(o["idx"][:kept], r["idx"][:kept]) and torch.equal(o["err"][:kept], r["err"][:kept])
    b.close()


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("dims", [(5000, 1, 1), (100, 41, 1), (33, 17, 9), (90, 91, 1)])
def test_padding_is_counted_without_a_copy(cuda, dims, mode):
    from fzgpumodules_b200 import kernels as K
    from fzgpumodules_b200._lib import check, lib
    x = _field(dims, 11, False) + np.float32(100)  # zeros widen the range (NOA)
    n = x.size
    total = (n + 4095) // 4096 * 4096 + (4096 if n % 8192 == 0 else 0)
    padded = np.zeros(total, np.float32)
    padded[:n] = x
    ref = K.lq_bs_rze_compress(torch.from_numpy(padded).to(cuda), dims, 1e-3, mode, 512, True, 0.5)
    d = torch.from_numpy(x).to(cuda)
    cap = K.max_outliers(total, 0.5)
    out = {k: torch.zeros_like(v) for k, v in ref.items() if k != "cap"}
    ws = K.Workspace()
    wp, wn = ws.get(total, d.device, cap)
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    f = lib().fzb_lq_bs_rze_compress_padded
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_uint64, C.c_uint64, C.c_void_p, C.c_float, C.c_int, C.c_float, C.c_uint32, C.c_int,
                  C.c_void_p, C.c_void_p, C.c_uint64, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p,
                  C.c_size_t, C.c_void_p]
    check(f(p(d), n, total, (C.c_uint32 * 3)(*dims), 1e-3, mode, 0.0, 512, 1, p(out["err"]), p(out["idx"]), cap,
            p(out["count"]), p(out["rze"]), p(out["rze_size"]), p(out["eb_state"]), wp, wn, None), "padded")
    torch.cuda.synchronize()
    size = int(ref["rze_size"].item())
    assert int(out["rze_size"].item()) == size and torch.equal(out["rze"][:size], ref["rze"][:size])
    assert torch.equal(out["eb_state"], ref["eb_state"])
    cnt = int(ref["count"].item())
    assert int(out["count"].item()) == cnt and torch.equal(out["idx"][:cnt], ref["idx"][:cnt])
    assert torch.equal(out["err"][:cnt], ref["err"][:cnt])
