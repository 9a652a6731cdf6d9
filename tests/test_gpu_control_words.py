"""A call clears the control words of its workspace itself, with and without a
value-base scan, for one and for several prepass blocks (1024 chunks each): the results
from a workspace full of set bits equal those from a zeroed one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class _Filled:
    """A workspace refilled with `byte` before every call that takes it."""

    def __init__(self, K, byte):
        self.ws, self.byte = K.Workspace(), byte

    def get(self, *a, **k):
        self.ws.get(*a, **k)
        self.ws.buf.fill_(self.byte)
        return self.ws.get(*a, **k)

    get_bytes = lambda self, need, dev: (self.ws.get_bytes(need, dev), self.ws.buf.fill_(self.byte))[0]
    status = lambda self: self.ws.status()


@pytest.mark.parametrize("dims", [(4000, 1, 1), (100, 41, 1), (64, 64, 64), (17, 9, 5), (8192 * 1025, 1, 1)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_chain_on_a_dirty_workspace(cuda, dims, mode):
    from fzgpumodules_b200 import kernels as K
    n = dims[0] * dims[1] * dims[2]
    x = 5.0 * torch.sin(0.01 * torch.arange(n, device=cuda))
    x += 0.01 * torch.randn(n, device=cuda, generator=torch.Generator(cuda).manual_seed(n))
    x[::97] = 20.0
    got = []
    for byte in (0, 255):
        ws = _Filled(K, byte)
        f = K.lq_bs_rze_compress(x, dims, 1e-2, mode, 40, True, 1.0, ws=ws)
        assert ws.status() == 0
        size, cnt = int(f["rze_size"].item()), int(f["count"].item())
        eb = float(f["eb_state"][1].item())
        y = K.lq_bs_rze_decompress(f["rze"], size, f["err"], f["idx"], f["count"], f["err"].numel(), n, dims, eb, True, ws=ws)
        assert ws.status() == 0
        raw = K.rze_decode(f["rze"][:size], 2 * n, ws=ws)
        p = K.pfpl_compress(x, 1e-3, mode, ws=ws)
        ps = int(p["rze_size"].item())
        z = K.pfpl_decompress(p["rze"], ps, p["vals"], p["idx"], p["count"], p["cap"], n, 1e-3, mode,
                              float(p["eb_state"][1].item()), ws=ws)
        got.append([f["rze"][:size], f["idx"][:cnt], y, raw, p["rze"][:ps], z])
    for a, b in zip(*got):
        assert torch.equal(a, b)
