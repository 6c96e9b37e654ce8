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
