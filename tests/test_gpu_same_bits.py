"""The register-resident kernels and the tcgen05 kernels give the same bits: a call whose scratch outputs are off the 16-byte
grid of bulk stores goes to the tcgen05 kernels, the same call on aligned buffers to the register-resident ones. So the result
of a shard does not depend on which kernels the whole call takes, and neither family can drift from the other unnoticed."""

import pytest
import torch

from tests.test_gpu_timeout import _backward, _buffers, _forward

pytestmark = pytest.mark.gpu

CELLS = ("lstm", "slstm", "gru", "elman")
WIDTHS = tuple(range(16, 257, 16))   # odd multiples of 16 from 80 on: 16-unit slices there, a half-filled last CTA here
# every width with every cell; batches: one row, a ragged second group, three groups
SHAPES = [(CELLS[j], (1, 9, 20)[(i + j) % 3], (1, 14, 33)[(i + 2 * j) % 3], 1 + (i + j) % 2, D) for i, D in enumerate(WIDTHS) for j in range(4)]
SHAPES += [("lstm", 150, 9, 6, 32), ("elman", 201, 5, 12, 48), ("lstm", 40, 6, 6, 112), ("slstm", 72, 5, 48, 16)]   # 16-row tiles on the tcgen05 side


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}-B{s[1]}-T{s[2]}-N{s[3]}-D{s[4]}")
def test_both_kernel_families_agree_bit_for_bit(shape, cuda_device):
    from flashrnn_b200 import _lib

    lib = _lib.load()
    cell, B, T, N, D = shape
    plan = _lib.plan(cell, B, T, N, D)
    no_backward = cell == "slstm" and (D in (208, 240) or (D == 16 and B > 40))   # the backward stays on tcgen05 either way
    assert _lib.register_kernels(cell, False, B, N, D) == (True, not no_backward)
    t = _buffers(_lib, cell, B, T, N, D, cuda_device)
    g = torch.Generator().manual_seed(5)
    t["dH"] = torch.randn(t["hist"].shape, generator=g).to(cuda_device)
    t["dC"] = torch.randn(t["carry"].shape, generator=g).to(cuda_device)
    err = torch.zeros(32, dtype=torch.int32, device=cuda_device)
    outs = {}
    for route in ("register", "tcgen05"):
        if route == "tcgen05":   # 8 bytes off: both families store these two in words of at most 4 bytes
            for k in ("hbf", "dgr"):
                t[k] = torch.zeros(t[k].numel() + 4, dtype=torch.bfloat16, device=cuda_device)[4:]
                assert t[k].data_ptr() % 16 == 8
        for k in ("hist", "carry", "cache", "dwx", "dinit", "dbp"):
            t[k].zero_()
        assert _forward(lib, _lib, cell, B, T, N, D, t, err, 0) == 0
        assert _backward(lib, _lib, cell, B, T, N, D, t, err, 0) == 0
        torch.cuda.synchronize()
        assert err[0].item() == 0, err[:3].tolist()
        outs[route] = {k: t[k].clone() for k in ("hist", "carry", "cache", "hbf", "dwx", "dgr", "dinit", "dbp")}
    for k, want in outs["tcgen05"].items():
        got = outs["register"][k]
        assert torch.isfinite(want.float() if want.dtype == torch.bfloat16 else want.to(torch.float64)).all(), (shape, k)
        if k == "dbp" and plan.batch_tile == 16:
            # 8 + 8 rows against 16 rows one by one: at most 15 roundings each of a partial sum of |row sums|
            rows = outs["tcgen05"]["dwx"].double().sum(dim=1).abs()                          # [B,GW,N,D], dWx = dG = what db sums
            rows = torch.nn.functional.pad(rows, (0, 0, 0, 0, 0, 0, 0, -B % 16)).unflatten(0, (-1, 16)).sum(dim=1).flatten()
            assert ((got.double() - want.double()).abs() <= 2 * 15 * 2.0 ** -24 * 1.01 * rows + 1e-30).all(), shape
        else:
            assert torch.equal(got.view(torch.uint8), want.view(torch.uint8)), (shape, k)


@pytest.mark.parametrize("D", [80, 208])
def test_multiples_of_sixteen_are_not_padded(D, cuda_device):
    """Results are dense, own their memory, and are those of a prepared sequence (which never pads) bit for bit."""
    from flashrnn_b200 import PreparedSequence, flashrnn_torch
    from flashrnn_b200.workloads import make_inputs

    wx, R, b, init = (t.to(cuda_device).contiguous() for t in make_inputs("lstm", 9, 11, 2, D, 78))
    history, carry = flashrnn_torch(wx.requires_grad_(True), R, b, init, cell="lstm", numerics="fp32_state_bf16_mma")
    assert history.is_contiguous() and carry.is_contiguous()
    assert history.untyped_storage().nbytes() == history.numel() * 4
    seq = PreparedSequence(wx.detach(), R, b, init, "lstm")
    out, final = seq.run()
    seq.check()
    assert torch.equal(out, history) and torch.equal(final, carry)
