"""Host side of the status word, with the word in host memory."""
import pytest
import torch

from return_b200.ext import ops

DEV = torch.device("cuda:0")


@pytest.fixture
def word(monkeypatch):
    t = torch.zeros(1, dtype=torch.int32)
    monkeypatch.setattr(ops, "_tc5_status", {DEV: t})
    monkeypatch.setattr(ops, "_tc5_launched", set())
    return t


def test_a_replay_marks_what_its_capture_saw(word):
    ops._tc5_launched.add(DEV)                                # something else ran before and was not looked at yet
    with ops.StatusWatch(DEV) as none:
        pass
    assert not none.waits and DEV in ops._tc5_launched
    with ops.StatusWatch(DEV) as some:
        ops._tc5_launched.add(DEV)
    assert some.waits
    ops.check_status(DEV)
    word.fill_(1)
    none.replayed()
    ops.check_status(DEV)                                     # no kernel with a wait ran: nobody asks
    some.replayed()
    with pytest.raises(ops.KernelError, match="bounded wait"):
        ops.check_status(DEV)
    assert int(word) == 0
    some.replayed()
    ops.check_status(DEV)


def test_the_word_that_comes_along(word):
    to = torch.zeros(1, dtype=torch.int32)
    word.fill_(1)
    assert not ops.copy_status(DEV, to)
    ops._tc5_launched.add(DEV)
    assert ops.copy_status(DEV, to) and int(to) == 1
    with pytest.raises(ops.KernelError):
        ops.raise_status(DEV, int(to))
    ops.raise_status(DEV, 0)
    assert int(word) == 0


def test_a_device_without_an_index_is_the_current_one(word, monkeypatch):
    monkeypatch.setattr(ops, "_device_index", lambda: 0)
    for ask in (lambda: ops.check_status("cuda"), lambda: ops.check_status(torch.device("cuda")), lambda: ops.raise_status("cuda", int(word))):
        ops._tc5_launched.add(DEV)
        word.fill_(1)
        with pytest.raises(ops.KernelError):
            ask()
        assert int(word) == 0
    to = torch.zeros(1, dtype=torch.int32)
    ops._tc5_launched.add(DEV)
    assert ops.copy_status("cuda", to)
    with ops.StatusWatch("cuda") as watch:
        ops._tc5_launched.add(DEV)
    assert watch.waits
