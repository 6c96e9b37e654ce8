"""Wide heads with R in registers against the tensor-memory kernels of the same split, bit for bit (see test_gpu_same_bits.py): every
split and chunk length of the two, ragged groups, and calls shorter than, as long as and longer than the 64 slots of the exchange."""

import pytest
import torch

from tests.test_gpu_timeout import _backward, _buffers, _forward

pytestmark = pytest.mark.gpu

# (cell, B, T, N, D), split of the contraction forward and backward, rows of a forward and a backward group: 0 = not one of these
# kernels, nothing to compare
CASES = [
    (("lstm", 1, 1, 1, 576), (4, 0), (8, 0)), (("gru", 9, 64, 1, 640), (2, 8), (8, 8)), (("slstm", 8, 65, 1, 640), (4, 8), (8, 8)),
    (("lstm", 16, 130, 1, 768), (2, 8), (8, 8)), (("slstm", 3, 130, 1, 768), (4, 8), (8, 8)), (("gru", 16, 33, 1, 768), (2, 8), (8, 8)),
    (("lstm", 11, 9, 1, 832), (2, 0), (8, 0)), (("lstm", 8, 97, 1, 896), (4, 8), (8, 8)), (("gru", 5, 200, 1, 1024), (4, 8), (8, 8)),
    (("elman", 16, 130, 1, 768), (2, 8), (8, 8)), (("lstm", 8, 66, 1, 1024), (4, 8), (8, 8)), (("lstm", 13, 7, 1, 1024), (2, 8), (8, 16)),
    (("slstm", 32, 5, 1, 1024), (2, 0), (16, 0)), (("slstm", 9, 4, 1, 960), (2, 0), (8, 0)), (("elman", 13, 67, 1, 1024), (2, 4), (8, 8)),
    (("elman", 9, 70, 1, 1536), (2, 4), (0, 8)), (("elman", 7, 5, 1, 1792), (2, 8), (0, 8)), (("slstm", 32, 70, 1, 896), (2, 4), (16, 0)),
    (("gru", 22, 16, 1, 1024), (2, 4), (16, 0)), (("gru", 30, 64, 1, 832), (2, 0), (16, 0)), (("gru", 30, 70, 1, 768), (2, 4), (16, 0)),
    (("elman", 30, 130, 1, 768), (2, 4), (16, 8)), (("elman", 64, 66, 1, 768), (0, 2), (0, 8)), (("gru", 16, 66, 1, 1280), (2, 8), (0, 16)),
]
OUT = {"forward": ("hist", "carry", "cache", "hbf"), "backward": ("dwx", "dgr", "dinit", "dbp")}


def _run(lib, _lib, shape, t, dev):
    err = torch.zeros(32, dtype=torch.int32, device=dev)
    cell, B, T, N, D = shape
    assert _forward(lib, _lib, cell, B, T, N, D, t, err, 0) == 0
    assert _backward(lib, _lib, cell, B, T, N, D, t, err, 0) == 0
    torch.cuda.synchronize()
    assert err[0].item() == 0, err[:3].tolist()
    return {k: t[k].clone() for names in OUT.values() for k in names}


def _shifted(x, elements):
    y = torch.empty(x.numel() + elements, dtype=x.dtype, device=x.device)[elements:].view(x.shape)
    return y.copy_(x)


@pytest.mark.parametrize("shape,splits,rows", CASES, ids=lambda v: "-".join(str(x) for x in v))
def test_wide_heads_agree_with_the_tensor_memory_kernels(shape, splits, rows, cuda_device):
    from flashrnn_b200 import _lib

    lib = _lib.load()
    plan = _lib.plan(*shape)
    cell, B, _, N, D = shape
    assert (plan.fwd_ksplit, plan.bwd_ksplit) == splits and _lib.register_rows(cell, False, B, N, D) == rows
    t = _buffers(_lib, *shape, cuda_device)
    g = torch.Generator().manual_seed(12)
    t["dH"] = torch.randn(t["hist"].shape, generator=g).to(cuda_device)
    t["dC"] = torch.randn(t["carry"].shape, generator=g).to(cuda_device)
    got = _run(lib, _lib, shape, t, cuda_device)
    for k in ("hbf",) * bool(rows[0]) + ("dwx",) * bool(rows[1]):   # 8 bytes off the grid of bulk stores, which the tensor-memory kernels do not use here
        t[k] = _shifted(torch.zeros_like(t[k]), 8 // t[k].element_size())
    for k in ("hist", "carry", "cache", "dgr", "dinit", "dbp"):
        t[k].zero_()
    want = _run(lib, _lib, shape, t, cuda_device)
    for k in OUT["forward"] * bool(rows[0]) + OUT["backward"] * bool(rows[1]):
        assert torch.equal(got[k].view(torch.uint8), want[k].view(torch.uint8)), (shape, k)


@pytest.mark.parametrize("shape", [("lstm", 8, 5, 2, 96), ("elman", 3, 4, 1, 160), ("gru", 8, 6, 1, 320)],
                         ids=lambda v: "-".join(str(x) for x in v))
def test_forward_fragments_from_r_off_the_16_byte_grid(shape, cuda_device):
    from flashrnn_b200 import _lib

    lib = _lib.load()
    t = _buffers(_lib, *shape, cuda_device)
    cell, B, T, N, D = shape
    assert _lib.register_rows(cell, False, B, N, D)[0] == 8   # the only kernels that take R off the grid
    err = torch.zeros(32, dtype=torch.int32, device=cuda_device)
    outs = []
    for R in (t["R"], _shifted(t["R"], 2)):
        t["R"] = R
        assert _forward(lib, _lib, cell, B, T, N, D, t, err, 0) == 0
        torch.cuda.synchronize()
        assert err[0].item() == 0
        outs.append([t[k].clone() for k in OUT["forward"]])
    for a, b in zip(*outs):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8)), shape
