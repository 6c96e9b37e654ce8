"""dR contraction of widths that are no multiple of 64 (boxes that reach past a head, several column tiles), of widths that no equal
whole-box tiles divide (320, 448, 640) and of sequences shorter than a chunk: against an fp64 einsum of the same bf16 operands."""

import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [("gru", 3, 70, 2, 80), ("lstm", 2, 33, 3, 48), ("elman", 5, 64, 1, 112), ("gru", 13, 100, 2, 208), ("lstm", 1, 1, 1, 240),
         ("slstm", 2, 65, 2, 176), ("lstm", 4, 40, 1, 320), ("elman", 3, 129, 2, 448), ("gru", 2, 63, 1, 640), ("lstm", 2, 64, 1, 704)]
# several batch rows to a chunk: a ragged last one, steps past the sequence, packed heads, every number of rows
CASES += [("lstm", 70, 1, 2, 80), ("gru", 33, 3, 1, 208), ("elman", 9, 32, 5, 32), ("lstm", 130, 2, 3, 64), ("slstm", 19, 7, 3, 16), ("gru", 5, 9, 1, 320)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-B{c[1]}-T{c[2]}-N{c[3]}-D{c[4]}")
def test_widths_that_do_not_fill_their_boxes(case, cuda_device):
    from flashrnn_b200 import _lib

    cell, B, T, N, D = case
    lib, plan = _lib.load(), _lib.plan(*case)
    gr, gb = plan.gates_r, plan.gates_b
    g = torch.Generator().manual_seed(D)
    dgr = torch.randn((B, T, gr, N, D), generator=g).to(cuda_device).bfloat16().contiguous()
    hbf = torch.randn((B, T + 1, N, D), generator=g).to(cuda_device).bfloat16().contiguous()
    db_part = torch.randn((plan.n_btiles, gb, N, D), generator=g).to(cuda_device)
    # a guard row on either side of the outputs
    dR = torch.full((gr * N * D * D + 2 * D,), float("nan"), device=cuda_device)
    db = torch.empty((gb, N, D), device=cuda_device)
    work = torch.full((max(plan.wgrad_work_bytes // 4, 1) + D,), float("nan"), device=cuda_device)
    err = torch.zeros(32, dtype=torch.int32, device=cuda_device)
    rc = lib.frnn_b200_wgrad(_lib.CELLS[cell], dgr.data_ptr(), hbf.data_ptr(), db_part.data_ptr(), dR[D:].data_ptr(), db.data_ptr(),
                             work.data_ptr(), B, T, N, D, err.data_ptr(), torch.cuda.current_stream(cuda_device).cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0 and err[0].item() == 0
    assert dR[:D].isnan().all() and dR[-D:].isnan().all() and work[-D:].isnan().all()
    ref = torch.einsum("btgno,btnp->gnop", dgr.double(), hbf[:, :T].double())
    mag = torch.einsum("btgno,btnp->gnop", dgr.double().abs(), hbf[:, :T].double().abs())
    # fp32 sums of exact products of bf16 values: one rounding per term of a partial sum of at most `mag`
    assert ((dR[D:-D].view(gr, N, D, D).double() - ref).abs() <= B * T * 2.0 ** -23 * mag).all()


@pytest.mark.parametrize("case", [("lstm", 3, 70, 2, 80), ("gru", 2, 5, 3, 32), ("lstm", 2, 33, 1, 128)], ids=lambda c: f"{c[0]}-B{c[1]}-T{c[2]}-N{c[3]}-D{c[4]}")
def test_last_hidden_state_belongs_to_no_product(case, cuda_device):
    """Slot T of bf16 h is not part of the sum, whatever stands there."""
    from flashrnn_b200 import _lib

    cell, B, T, N, D = case
    lib, plan = _lib.load(), _lib.plan(*case)
    gr, gb = plan.gates_r, plan.gates_b
    g = torch.Generator().manual_seed(3)
    dgr = torch.randn((B, T, gr, N, D), generator=g).to(cuda_device).bfloat16()
    hbf = torch.randn((B, T + 1, N, D), generator=g).to(cuda_device).bfloat16()
    db_part = torch.zeros((plan.n_btiles, gb, N, D), device=cuda_device)
    db, work = torch.empty((gb, N, D), device=cuda_device), torch.empty(max(plan.wgrad_work_bytes // 4, 1), device=cuda_device)
    err = torch.zeros(32, dtype=torch.int32, device=cuda_device)
    outs = []
    for last in (0.0, float("inf"), float("nan")):
        hbf[:, T] = last
        dR = torch.empty((gr, N, D, D), device=cuda_device)
        rc = lib.frnn_b200_wgrad(_lib.CELLS[cell], dgr.data_ptr(), hbf.data_ptr(), db_part.data_ptr(), dR.data_ptr(), db.data_ptr(),
                                 work.data_ptr(), B, T, N, D, err.data_ptr(), torch.cuda.current_stream(cuda_device).cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0 and err[0].item() == 0
        outs.append(dR)
    assert outs[0].isfinite().all() and torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
