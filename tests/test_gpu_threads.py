"""Host threads that call the library at once: a kernel's shared-memory limit must not be what one thread's call needs."""

import threading

import pytest
import torch

from tests.test_gpu_timeout import _backward, _buffers, _forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,D", [("lstm", 256), ("slstm", 128), ("gru", 48)])
def test_inference_and_training_threads_do_not_refuse_each_other(cell, D, cuda_device):
    """bf16 inference (small stages) in some threads, fp32 training of the same width (large ones) in others, each on its own
    stream and buffers: every launch is accepted and every result is that of a call made alone."""
    from flashrnn_b200 import _lib

    lib = _lib.load()
    B, T, N = 3, 2, 1
    zero_word = torch.zeros(1, dtype=torch.int32, device=cuda_device)

    class Caller:
        def __init__(self, train):
            self.train, self.t, self.refused = train, _buffers(_lib, cell, B, T, N, D, cuda_device), []
            if not train:
                self.t["wx"] = self.t["wx"].bfloat16()
            self.err = torch.zeros(32, dtype=torch.int32, device=cuda_device)
            self.stream = torch.cuda.Stream(cuda_device)

        def launches(self):
            """(function, arguments) of one pass, made once: the less Python between two calls, the more they overlap."""
            t, made = self.t, []

            class Recorder:
                def __getattr__(self, name):
                    fn = getattr(lib, name)
                    return lambda *args: made.append((fn, tuple(k(v) for k, v in zip(fn.argtypes, args)))) or 0

            with torch.cuda.stream(self.stream):
                if self.train:
                    _forward(Recorder(), _lib, cell, B, T, N, D, t, self.err, 0)
                    _backward(Recorder(), _lib, cell, B, T, N, D, t, self.err, 0)
                else:
                    Recorder().frnn_b200_forward_prepared(
                        _lib.CELLS[cell], t["wx"].data_ptr(), 1, t["R"].data_ptr(), t["b"].data_ptr(), t["init"].data_ptr(),
                        t["hist"].data_ptr(), t["carry"].data_ptr(), None, B, T, N, D, 1, zero_word.data_ptr(), 0,
                        self.err.data_ptr(), self.stream.cuda_stream)
            return made

        def run(self, calls):
            made = self.launches()
            torch.ones(1, device=cuda_device)   # a new thread has no current CUDA context before its first runtime call
            for _ in range(calls):
                for fn, args in made:
                    rc = fn(*args)
                    if rc:
                        self.refused.append(rc)

        def results(self):
            keys = ("hist", "carry", "dwx", "dinit") if self.train else ("hist", "carry")
            return [self.t[k].clone() for k in keys]

    callers = [Caller(train=i % 2 == 0) for i in range(8)]
    torch.cuda.synchronize()
    for c in callers:
        c.run(1)
    torch.cuda.synchronize()
    alone = [c.results() for c in callers]
    threads = [threading.Thread(target=c.run, args=(4000,)) for c in callers]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not [(c.train, c.refused[:3]) for c in callers if c.refused]
    for c, want in zip(callers, alone):
        assert c.err[0].item() == 0
        for got, w in zip(c.results(), want):
            assert torch.equal(got, w)


def test_threads_with_other_widths_do_not_refuse_each_other(cuda_device):
    """dR of 64-column and of 256-column tiles, and tensor-memory recurrences of 288 and of 512 units (one kernel each, with different
    amounts of shared memory): every launch is accepted."""
    from flashrnn_b200 import _lib

    lib = _lib.load()

    class Caller:
        def __init__(self, D, wgrad):
            self.refused, self.stream, self.err = [], torch.cuda.Stream(cuda_device), torch.zeros(32, dtype=torch.int32, device=cuda_device)
            t = self.t = _buffers(_lib, "lstm", 2, 2, 1, D, cuda_device)
            plan = _lib.plan("lstm", 2, 2, 1, D)
            if not wgrad:   # 8 bytes off the grid of bulk stores, which the kernels with R in registers use
                for k in ("hbf", "dgr"):
                    t[k] = torch.zeros(t[k].numel() + 4, dtype=torch.bfloat16, device=cuda_device)[4:]
            self.dR, self.db = torch.zeros((4, 1, D, D), device=cuda_device), torch.zeros((4, 1, D), device=cuda_device)
            self.work = torch.zeros(max(plan.wgrad_work_bytes // 4, 1), device=cuda_device)
            made = []

            class Recorder:
                def __getattr__(self, name):
                    fn = getattr(lib, name)
                    return lambda *args: made.append((fn, tuple(k(v) for k, v in zip(fn.argtypes, args)))) or 0

            with torch.cuda.stream(self.stream):
                if wgrad:
                    Recorder().frnn_b200_wgrad(_lib.CELLS["lstm"], t["dgr"].data_ptr(), t["hbf"].data_ptr(), t["dbp"].data_ptr(), self.dR.data_ptr(),
                                               self.db.data_ptr(), self.work.data_ptr(), 2, 2, 1, D, self.err.data_ptr(), self.stream.cuda_stream)
                else:
                    _forward(Recorder(), _lib, "lstm", 2, 2, 1, D, t, self.err, 0)
                    _backward(Recorder(), _lib, "lstm", 2, 2, 1, D, t, self.err, 0)
            self.made = made

        def run(self, calls):
            torch.ones(1, device=cuda_device)   # a new thread has no current CUDA context before its first runtime call
            for _ in range(calls):
                self.refused += [rc for rc in (fn(*args) for fn, args in self.made) if rc]

    for widths, wgrad in (((64, 256), True), ((288, 512), False)):
        callers = [Caller(widths[i % 2], wgrad) for i in range(6)]
        torch.cuda.synchronize()
        threads = [threading.Thread(target=c.run, args=(2000,)) for c in callers]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        torch.cuda.synchronize()
        assert not [(widths[i % 2], c.refused[:3]) for i, c in enumerate(callers) if c.refused]
        assert all(c.err[0].item() == 0 for c in callers)
