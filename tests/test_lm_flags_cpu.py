"""CPU: what the LM's error flags are called."""
import re
from pathlib import Path

import pytest

HEADER = Path(__file__).resolve().parent.parent / "include" / "moshi_b200.h"


@pytest.mark.parametrize("flag,word", [("TOKEN_RANGE", "embedding table"), ("CODE_RANGE", "codebook"), ("KV_CAPACITY", "ring"), ("WAIT", "wait")])
def test_every_flag_has_its_own_words(flag, word):
    from moshi_b200 import _lib
    value = int(re.search(rf"#define B200_FLAG_{flag} (\d+)", HEADER.read_text()).group(1))
    text = _lib.lib().b200_lm_flag_text(value).decode()
    assert word in text
    others = {"embedding table", "codebook", "ring", "wait"} - {word}
    assert not any(o in text for o in others), text


def test_no_flag_no_words_and_the_gravest_first():
    from moshi_b200 import _lib
    lib = _lib.lib()
    assert lib.b200_lm_flag_text(0) == b""
    assert b"wait" in lib.b200_lm_flag_text(15)
    assert lib.b200_lm_flag_text(64) != b""


def test_a_handle_without_a_stream_has_nothing_to_report():
    from moshi_b200 import _lib
    assert _lib.lib().b200_lm_check_waits(None) == 0
