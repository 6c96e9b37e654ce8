"""Groups of 16 and 24 batch rows and heads of 288 to 512 units of the register-resident kernels, against the tcgen05 kernels bit for
bit (see test_gpu_same_bits.py), at the edges of their rules: the smallest and largest batch of each group size, ragged last groups,
the first and last width of each instantiation, every length of a last transfer (4 steps, fewer where shared memory is short)."""

import pytest
import torch

from tests.test_gpu_timeout import _backward, _buffers, _forward

pytestmark = pytest.mark.gpu

# (cell, B, T, N, D), rows of a forward and a backward group: 0 = tcgen05
CASES = [
    (("lstm", 3, 9, 1, 288), (8, 8)), (("slstm", 8, 5, 1, 320), (8, 8)), (("gru", 9, 6, 1, 384), (8, 8)), (("elman", 1, 7, 2, 416), (8, 8)),
    (("lstm", 9, 4, 1, 512), (8, 8)), (("slstm", 2, 3, 1, 512), (8, 8)), (("gru", 1, 1, 1, 480), (8, 8)), (("elman", 17, 2, 1, 512), (8, 8)),
    (("lstm", 256, 5, 4, 128), (16, 16)), (("gru", 97, 4, 11, 96), (16, 16)), (("slstm", 155, 3, 8, 64), (16, 16)),
    (("elman", 266, 6, 4, 128), (16, 16)), (("lstm", 57, 7, 4, 160), (16, 16)), (("gru", 64, 3, 3, 256), (16, 16)),
    (("lstm", 64, 2, 1, 384), (16, 16)), (("gru", 57, 5, 1, 448), (0, 16)), (("slstm", 64, 3, 1, 512), (16, 0)), (("lstm", 200, 4, 4, 112), (16, 16)),
    (("lstm", 84, 5, 3, 256), (24, 24)), (("gru", 100, 3, 3, 240), (24, 0)), (("slstm", 90, 2, 3, 224), (24, 24)), (("elman", 720, 2, 1, 256), (24, 24)),
    # one more CTA on the SM: the first batch that needs it, many heads of few rows; the other side of the rules for wider groups
    (("lstm", 3, 5, 34, 144), (8, 0)), (("slstm", 8, 3, 30, 160), (8, 0)), (("gru", 1, 4, 30, 144), (8, 0)),
    (("lstm", 304, 5, 8, 32), (8, 8)), (("slstm", 310, 3, 8, 32), (8, 8)), (("lstm", 304, 6, 4, 64), (8, 16)), (("slstm", 301, 3, 4, 64), (16, 16)),
    (("gru", 304, 5, 4, 64), (8, 16)), (("elman", 304, 3, 1, 224), (8, 16)), (("lstm", 112, 3, 1, 512), (16, 0)), (("slstm", 64, 3, 1, 384), (16, 16)),
    (("lstm", 22, 3, 4, 384), (0, 0)),
    (("lstm", 64, 3, 2, 384), (0, 24)), (("elman", 96, 2, 3, 512), (24, 0)), (("lstm", 152, 3, 3, 256), (0, 0)),
]


@pytest.mark.parametrize("shape,rows", CASES, ids=lambda v: "-".join(str(x) for x in v))
def test_wider_groups_and_heads_agree_with_the_tcgen05_kernels(shape, rows, cuda_device):
    from flashrnn_b200 import _lib

    lib = _lib.load()
    cell, B, T, N, D = shape
    assert _lib.register_rows(cell, False, B, N, D) == rows
    t = _buffers(_lib, cell, B, T, N, D, cuda_device)
    g = torch.Generator().manual_seed(11)
    t["dH"] = torch.randn(t["hist"].shape, generator=g).to(cuda_device)
    t["dC"] = torch.randn(t["carry"].shape, generator=g).to(cuda_device)
    err = torch.zeros(32, dtype=torch.int32, device=cuda_device)
    outs = {}
    for route in ("register", "tcgen05"):
        if route == "tcgen05":   # 8 bytes off the grid of bulk stores
            for k in ("hbf", "dgr"):
                t[k] = torch.zeros(t[k].numel() + 4, dtype=torch.bfloat16, device=cuda_device)[4:]
        for k in ("hist", "carry", "cache", "dwx", "dinit", "dbp"):
            t[k].zero_()
        assert _forward(lib, _lib, cell, B, T, N, D, t, err, 0) == 0
        assert _backward(lib, _lib, cell, B, T, N, D, t, err, 0) == 0
        torch.cuda.synchronize()
        assert err[0].item() == 0, err[:3].tolist()
        outs[route] = {k: t[k].clone() for k in ("hist", "carry", "cache", "hbf", "dwx", "dgr", "dinit", "dbp")}
    plan = _lib.plan(cell, B, T, N, D)
    for k, want in outs["tcgen05"].items():
        got = outs["register"][k]
        if k == "dbp" and plan.batch_tile == 16 and rows[1] in (8, 24):
            # halves of 8 rows against 16 rows one by one: at most 15 roundings each of a partial sum of |row sums|
            s = outs["tcgen05"]["dwx"].double().sum(dim=1).abs()
            s = torch.nn.functional.pad(s, (0, 0, 0, 0, 0, 0, 0, -B % 16)).unflatten(0, (-1, 16)).sum(dim=1)
            if cell == "gru":   # four bias gradients from three gate gradients; the candidate's recurrent one is at most its input one
                s = torch.cat((s[:, 2:3], s), dim=1)
            assert ((got.double() - want.double()).abs() <= 2 * 15 * 2.0 ** -24 * 1.01 * s.flatten() + 1e-30).all(), shape
        else:
            assert torch.equal(got.view(torch.uint8), want.view(torch.uint8)), (shape, k)
