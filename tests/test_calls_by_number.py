"""Calls with packed arguments: the library and ``_lib`` agree on the functions, their arguments and the words' order."""

import pytest

from moonep_b200.ops import _lib


@pytest.mark.parametrize("name", _lib._BY_NUMBER)
def test_argument_counts(name):
    _lib.caller(name)  # compares the library's count with the signature's


def test_words_arrive_in_order():
    # sizes that the function refuses before it looks at a device: the message tells which argument it saw
    call = _lib.caller("moonep_grouped_gemm_pair")
    ok = dict(x=0, w0=0, w1=0, out=0, row_scale=0, cu=0, G=2, rows=128, K=64, n=256, mode=0, status=0, ms=1 << 40, sms=0,
              group_map=0, w_slots=0, pre_gate=0, pre_up=0, stream=0)  # fmt: skip
    for change, message in (({"K": 65}, "K must be"), ({"n": 255}, "N per group must be a multiple of 256"),
                            ({"mode": 1, "n": 100}, "multiple of 128"), ({"mode": 1}, "needs the up-projection"),
                            ({"pre_up": 16}, "go together"), ({"pre_gate": 16}, "go together")):  # fmt: skip
        assert call(*(ok | change).values()) != 0
        assert message in _lib.load().moonep_last_error().decode()


def test_unknown_number():
    assert _lib.load().moonep_call(len(_lib._BY_NUMBER), None) == -1
