"""The device word in which kernels record that a bounded wait ran out."""
import os
import re

import pytest
import torch

from burn_lm_b200 import kernels as K
from burn_lm_b200.csrc import build


@pytest.fixture
def words(monkeypatch):
    """A table of its own, whose words lie in host memory."""
    monkeypatch.setattr(K, "_status", {})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    zeros = torch.zeros
    monkeypatch.setattr(torch, "zeros", lambda *size, dtype, device: zeros(*size, dtype=dtype))
    return K._status


SPELLINGS = [torch.device("cuda:1"), "cuda:1", 1, "cuda", torch.device("cuda"), torch.device("cuda", 1), torch.device(1)]


@pytest.mark.parametrize("first", range(len(SPELLINGS)))
def test_every_spelling_of_a_device_names_one_word(words, first):
    word = K.status_word(SPELLINGS[first])
    for device in SPELLINGS:
        assert K.status_word(device) is word
    assert K.status_word("cuda:0") is not word and K.status_word(torch.device("cuda:1")) is word
    assert len(words) == 2


def test_a_wait_that_ran_out_is_reported_once_by_any_spelling(words):
    for device in SPELLINGS:
        K.status_word(torch.device("cuda:1")).fill_(11)
        with pytest.raises(K.KernelError):
            K.check_status(device)
        assert K.check_status("cuda:1") is None


def test_every_code_has_a_message_and_is_one_files_own():
    text = {name: open(os.path.join(build.HERE, name)).read() for name in sorted({f for m in build.MODULES.values() for f in m} | set(build.HEADERS))}
    codes = {name: int(n) for t in text.values() for name, n in re.findall(r"(\w+_TIMEOUT_\w+) = (\d+)", t)}
    assert len(set(codes.values())) == len(codes) > 10
    for name, code in codes.items():
        assert code in K._WAITS, name
        assert len([f for f, t in text.items() if re.search(rf"\b{name}\b(?! =)", t)]) == 1, name
