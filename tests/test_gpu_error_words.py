"""Error words of eager launches, handed out in blocks and read back together: each launch's word is found under its name, across
blocks, threads and streams; a word that is out but not tracked yet is left alone; a refused launch's word is used again."""

import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def drained(cuda_device):
    from flashrnn_b200 import functional as F

    F.poll_errors(block=True)
    yield
    F._pending_errors.clear()
    F._blocks.clear()


def test_a_reported_word_is_found_under_its_name(cuda_device):
    from flashrnn_b200 import functional as F

    dev = torch.device("cuda", torch.cuda.current_device())
    size = F._ErrorBlock.SIZE
    words = []
    for i in range(2 * size + 3):                      # three blocks
        words.append(F._error_word(dev))
        F._track(words[-1], f"launch {i}")
    assert len({w.data_ptr() for w in words}) == len(words) and all(w.numel() == 32 for w in words)
    assert not any(w.any().item() for w in words)
    words[size + 5][:3] = torch.tensor([101, 7, 3], dtype=torch.int32, device=dev)
    with pytest.raises(RuntimeError, match=f"launch {size + 5}: .*code 101.*step 7, CTA 3"):
        F.poll_errors(block=True)
    F.poll_errors(block=True)                          # what is left is fine
    assert not F._pending_errors and not F._blocks


def test_words_on_the_way_are_left_for_the_next_time(cuda_device):
    from flashrnn_b200 import functional as F

    dev = torch.device("cuda", torch.cuda.current_device())
    F._track(F._error_word(dev), "before")
    word = F._error_word(dev)                          # its launch is just being made
    F.poll_errors(block=True)
    assert len(F._blocks) == 1
    word[0] = 106
    F._track(word, "late")
    with pytest.raises(RuntimeError, match="late: .*code 106"):
        F.poll_errors(block=True)
    # a launch that is refused never tracks its word: the next launch gets it
    refused = F._error_word(dev)
    assert F._error_word(dev).data_ptr() == refused.data_ptr()


def test_threads_and_streams_have_blocks_of_their_own(cuda_device):
    from flashrnn_b200 import functional as F

    dev = torch.device("cuda", torch.cuda.current_device())
    words, errors = [], []

    def work(name):
        try:
            with torch.cuda.stream(torch.cuda.Stream(dev)):
                for i in range(50):
                    w = F._error_word(dev)
                    words.append(w)
                    if i == 30 and name == "c":
                        w[0] = 103
                    F._track(w, f"{name}{i}")
        except Exception as e:  # pragma: no cover - reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(n,)) for n in "abcd"]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and len({w.data_ptr() for w in words}) == 200
    with pytest.raises(RuntimeError, match="c30: .*code 103"):
        F.poll_errors(block=True)


def test_word_of_a_backward_whose_contraction_was_refused(cuda_device, monkeypatch):
    """The recurrence runs with the word, so no later launch may get it, and what it reports is found."""
    from flashrnn_b200 import _lib, flashrnn_torch
    from flashrnn_b200 import functional as F
    from flashrnn_b200.workloads import make_inputs

    lib = _lib.load()

    class Refuses:
        def __getattr__(self, name):
            return (lambda *args: -2) if name == "frnn_b200_wgrad" else getattr(lib, name)

    given, inner = [], F._error_word
    monkeypatch.setattr(F, "_error_word", lambda device: given.append(inner(device)) or given[-1])
    wx, R, b, init = (t.to(cuda_device).requires_grad_(True) for t in make_inputs("lstm", 2, 3, 1, 64, 5))
    history, _ = flashrnn_torch(wx, R, b, init, cell="lstm", numerics="fp32_state_bf16_mma")
    monkeypatch.setattr(_lib, "load", Refuses)
    with pytest.raises(RuntimeError, match="frnn_b200_wgrad failed"):
        F._Recurrence._backward(history.grad_fn, torch.ones_like(history), None)
    assert len(given) == 2                             # forward, backward
    later = inner(torch.device("cuda", torch.cuda.current_device()))
    assert later.data_ptr() not in [w.data_ptr() for w in given]
    F._track(later, "later")
    given[1][0] = 106
    with pytest.raises(RuntimeError, match="frnn_b200_backward: .*code 106"):
        F.poll_errors(block=True)
