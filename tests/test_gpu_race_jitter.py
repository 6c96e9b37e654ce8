"""Race verification by delay injection: with err[6] = seed the kernels stall, in a quarter of the steps and for up
to 8 us, the epilogue warps, the tensor-core warp or the I/O warp of pseudo-randomly chosen CTAs, so that the CTAs of a group (and
the warp roles inside a CTA) drift against each other at every hand-off of the exchange protocols (operand pushes,
partial sums, staged stores, slot reuse). Every result must stay bit-identical to the undisturbed run. The hook is
compiled into the fp32-Wx instantiations of the kernels (the exchange code is the same for both Wx types).

The reference verifies its persistent kernels the same way (tools/race_verify.py: seeded 0-65 us delays plus a content
check of every exchanged operand).

With err[7] = 1 as well only the I/O warps are late, and the register-resident kernels run the loops that calls without hooks run (any
other hook selects a loop of its own); copies on another stream take bandwidth from the launches meanwhile."""

import pytest
import torch

from tests.test_gpu_timeout import _backward, _buffers, _forward

pytestmark = pytest.mark.gpu

# ((cell, B, T, N, D), batch rows of a forward and a backward group of the kernels with R in registers; 0: in tensor memory)
CASES = [
    # R in registers: one CTA per head, two staged tiles per CTA; clusters, a half-filled last CTA; groups of 16 and 24 rows
    (("lstm", 24, 20, 2, 48), (8, 8)), (("slstm", 9, 24, 2, 48), (8, 8)), (("lstm", 9, 24, 2, 48), (8, 8)), (("gru", 5, 33, 3, 32), (8, 8)),
    (("elman", 3, 40, 2, 16), (8, 8)), (("lstm", 9, 24, 2, 80), (8, 8)), (("gru", 8, 24, 1, 240), (8, 8)), (("lstm", 8, 40, 3, 256), (8, 8)),
    (("gru", 5, 33, 2, 128), (8, 8)), (("slstm", 16, 24, 4, 128), (8, 8)), (("elman", 9, 30, 1, 512), (8, 8)), (("lstm", 8, 22, 1, 512), (8, 8)),
    (("lstm", 200, 16, 4, 128), (16, 16)), (("lstm", 84, 12, 3, 256), (24, 24)), (("lstm", 304, 10, 8, 32), (8, 8)),
    # wide heads: shorter than the 64 slots of the exchange, and slots refilled and used again (from 65 steps on), for every split
    (("gru", 8, 16, 1, 768), (8, 8)), (("lstm", 16, 16, 1, 1024), (8, 16)), (("lstm", 4, 140, 1, 768), (8, 8)), (("gru", 16, 140, 1, 768), (8, 8)),
    (("lstm", 13, 132, 1, 1024), (8, 16)), (("elman", 30, 140, 1, 768), (16, 8)), (("slstm", 32, 131, 1, 896), (16, 0)),
    # R in tensor memory: clusters of 16- and 32-unit slices, 8- and 16-row tiles; the contraction split inside clusters; one CTA per
    # unit slice and the 1-D backward over global memory
    (("lstm", 200, 8, 6, 112), (0, 0)), (("gru", 57, 10, 1, 448), (0, 16)), (("slstm", 64, 10, 1, 512), (16, 0)), (("lstm", 152, 6, 3, 256), (0, 0)),
    (("lstm", 120, 8, 1, 512), (0, 0)), (("lstm", 8, 16, 1, 1280), (0, 0)), (("lstm", 16, 12, 1, 1280), (0, 0)), (("lstm", 4, 24, 1, 576), (8, 0)),
    (("lstm", 64, 12, 1, 768), (0, 0)),
]
OUTPUTS_FWD = ("hist", "carry", "cache", "hbf")
OUTPUTS_BWD = ("dwx", "dgr", "dinit", "dbp")


@pytest.mark.parametrize("shape,rows", CASES, ids=lambda v: "-".join(str(x) for x in v))
def test_results_do_not_depend_on_injected_delays(shape, rows, cuda_device):
    from flashrnn_b200 import _lib

    lib = _lib.load()
    cell, B, T, N, D = shape
    assert _lib.register_rows(cell, False, B, N, D) == rows
    t = _buffers(_lib, cell, B, T, N, D, cuda_device)
    t["dH"] = torch.randn(t["hist"].shape, generator=torch.Generator().manual_seed(3)).to(cuda_device)
    err = torch.zeros(32, dtype=torch.int32, device=cuda_device)

    def run(seed, io_only=0):
        err.zero_()
        err[6], err[7] = seed, io_only
        assert _forward(lib, _lib, cell, B, T, N, D, t, err, 0) == 0
        torch.cuda.synchronize()
        assert err[0].item() == 0, err[:3].tolist()
        fwd = {k: t[k].clone() for k in OUTPUTS_FWD}
        err.zero_()
        err[6], err[7] = seed, io_only
        assert _backward(lib, _lib, cell, B, T, N, D, t, err, 0) == 0
        torch.cuda.synchronize()
        assert err[0].item() == 0, err[:3].tolist()
        return {**fwd, **{k: t[k].clone() for k in OUTPUTS_BWD}}

    def same(a, b):   # bit patterns (the gate cache is raw bytes, NaNs cannot occur in the rest)
        return torch.equal(a.view(torch.uint8).flatten(), b.view(torch.uint8).flatten())

    calm = run(0)
    for seed in (1, 77, 4242):
        shaken = run(seed)
        for key, want in calm.items():
            assert same(shaken[key], want), (shape, seed, key)
    if rows == (0, 0):
        return
    # the loops of a call without hooks: late I/O warps, and another stream's copies between and during the launches
    noise, side = torch.empty(2, 1 << 24, device=cuda_device), torch.cuda.Stream(cuda_device)
    for seed in (9, 640):
        with torch.cuda.stream(side):
            for _ in range(40):
                noise[1].copy_(noise[0])
        shaken = run(seed, io_only=1)
        for key, want in calm.items():
            assert same(shaken[key], want), (shape, seed, key, "I/O")
    side.synchronize()


@pytest.mark.parametrize("case", [("lstm", 8, 20, 1024, 4, 0, 0), ("gru", 5, 16, 512, 2, 0, 0), ("lstm", 6, 12, 2048, 1, 0, 0),
                                  ("lstm", 4, 10, 2048, 2, 128, 3)],
                         ids=lambda c: f"{c[0]}-B{c[1]}-T{c[2]}-D{c[3]}-P{c[4]}-kt{c[5]}")
def test_wide_head_results_do_not_depend_on_injected_delays(case, cuda_device):
    """The row-sharded kernels (all ranks as one launch): write-once history slots, cluster K reduction, staged publication."""
    from flashrnn_b200 import poll_errors
    from flashrnn_b200.wide_head import WideHead
    from tests.test_gpu_wide_head import _inputs

    cell, B, T, D, P, kt, rs = case
    wx, R, b, init, d_history, d_carry = _inputs(cell, B, T, D, 31)
    # fp32 Wx: the hook is compiled into those instantiations (the exchange code does not depend on the Wx type)
    head = WideHead(cell, B, T, D, emulate_ranks=P, device=cuda_device, wx_dtype=torch.float32, k_tmem_max=kt,
                    ring_stages_max=rs, wait_limit_ms=3000)
    try:
        def run(seed):
            head.jitter = seed
            leaves = [x.to(cuda_device).requires_grad_(True) for x in (wx, R, b, init)]
            h, c = head(*leaves)
            ((h * d_history.to(cuda_device)).sum() + (c * d_carry.to(cuda_device)).sum()).backward()
            torch.cuda.synchronize()
            poll_errors(block=True)
            return [h.detach().clone(), c.detach().clone()] + [x.grad.clone() for x in leaves]

        calm = run(0)
        for seed in (5, 909):
            for got, want in zip(run(seed), calm):
                assert torch.equal(got, want), (case, seed)
    finally:
        head.close()
