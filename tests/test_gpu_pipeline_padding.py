"""Inputs whose size the pipeline pads, at any place in memory: the container is
that of the same values at an aligned address, and decodes to them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pipeline(chain, n, dims, mode):
    from fzgpumodules_b200 import pipeline as P
    pl = P.Pipeline(4 * n, P.PREALLOCATE)
    pl.setDims(*dims)
    if chain == "lq":
        a = pl.addStage(P.LorenzoQuantStage(1e-3, 512, 0.5, mode, True))
        b = pl.addStage(P.BitshuffleStage(16384, 2))
    else:
        a = pl.addStage(P.QuantizerStage(1e-3, mode, 32768, 0.5, code_bytes=4, zigzag_codes=True))
        d = pl.addStage(P.DifferenceStage(P.INT32, P.UINT32, 16384))
        b = pl.addStage(P.BitshuffleStage(16384, 2))
    c = pl.addStage(P.RZEStage(16384, 4))
    if chain == "lq":
        pl.connect(b, a, "codes")
    else:
        pl.connect(d, a, "codes")
        pl.connect(b, d)
    pl.connect(c, b)
    pl.finalize()
    assert pl.isFused()
    return pl


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("chain,dims", [("lq", (10007, 1, 1)), ("lq", (101, 99, 1)), ("lq", (33, 17, 9)),
                                        ("pfpl", (10007, 1, 1)), ("pfpl", (4095, 1, 1))])
def test_any_address(cuda, chain, dims, mode):
    n = int(np.prod(dims))
    rng = np.random.default_rng(n + mode)
    x = (np.cumsum(rng.normal(0, 0.02, n)) + 50).astype(np.float32)
    x[rng.integers(0, n, 20)] = 3000.0
    ref = None
    for shift in (0, 4, 8, 12, 1, 2, 3):
        room = torch.zeros(4 * n + 16, dtype=torch.uint8, device=cuda)
        room[shift:shift + 4 * n] = torch.from_numpy(x.view(np.uint8)).to(cuda)
        pl = _pipeline(chain, n, dims, mode)
        comp = pl.compress(room[shift:shift + 4 * n]).clone()
        if ref is None:
            ref = comp
            back = pl.decompress(comp)[:n].cpu().numpy()
            bound = 1e-3 * (np.abs(x) if chain == "pfpl" and mode == 1 else [1, np.abs(x).max(), np.ptp(x)][mode])
            # the pads' zeros widen a NOA range
            bound = np.maximum(bound, 1e-3 * np.abs(x).max()) if mode == 2 else bound
            assert (np.abs(back.astype(np.float64) - x) <= bound * (1 + 1e-5) + 4e-4).all()
        assert torch.equal(comp, ref), shift


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 4095, 4096, 10007, 4096 * 5 + 16])
def test_pfpl_padding_is_counted_without_a_copy(cuda, n, mode):
    import ctypes as C

    from fzgpumodules_b200 import kernels as K
    from fzgpumodules_b200._lib import check, lib
    rng = np.random.default_rng(n)
    x = (rng.normal(0, 1, n) + 100).astype(np.float32)  # zeros widen the range (NOA)
    x[rng.integers(0, n, max(1, n // 50))] = 1e6
    total = n // 4096 * 4096 + 2 * 4096
    padded = np.zeros(total, np.float32)
    padded[:n] = x
    ref = K.pfpl_compress(torch.from_numpy(padded).to(cuda), 1e-3, mode, 512, True, 1.0)
    d = torch.from_numpy(x).to(cuda)
    out = {k: torch.zeros_like(v) for k, v in ref.items() if k != "cap"}
    cap = ref["cap"]
    need = lib().fzb_pfpl_workspace_bytes(total, cap)
    work = torch.full((need,), 0xff, dtype=torch.uint8, device=cuda)
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    f = lib().fzb_pfpl_compress_padded
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_uint64, C.c_uint64, C.c_float, C.c_int, C.c_float, C.c_uint32, C.c_int, C.c_float,
                  C.c_void_p, C.c_void_p, C.c_uint64, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p,
                  C.c_size_t, C.c_void_p]
    check(f(p(d), n, total, 1e-3, mode, 0.0, 512, 1, float("inf"), p(out["vals"]), p(out["idx"]), cap, p(out["count"]),
            p(out["rze"]), p(out["rze_size"]), p(out["eb_state"]), p(work), need, None), "padded")
    torch.cuda.synchronize()
    size, cnt = int(ref["rze_size"].item()), int(ref["count"].item())
    assert int(out["rze_size"].item()) == size and torch.equal(out["rze"][:size], ref["rze"][:size])
    assert torch.equal(out["eb_state"], ref["eb_state"])
    assert int(out["count"].item()) == cnt and torch.equal(out["idx"][:cnt], ref["idx"][:cnt])
    assert torch.equal(out["vals"][:cnt], ref["vals"][:cnt])
