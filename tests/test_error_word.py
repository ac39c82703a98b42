"""Every kernel that reports a bounded wait is handed the error word that ends its
call, the self-test of the waits too: what the self-test shows then holds for the
pair kernels."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "entropical_gb300" / "csrc"


def calls(text, name):
    """The argument texts of every call of name."""
    for m in re.finditer(rf"\b{name}\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


def test_the_self_test_shares_the_pair_kernels_error_word():
    text = (CSRC / "api.cu").read_text()
    word = {name: [re.findall(r"&c(?:->|\.)(\w+->\w+|\w+)", a) for a in calls(text, name)]
            for name in ("launch_density", "launch_density_sym", "launch_wait_test")}
    assert all(word.values())
    for name, found in word.items():
        assert all(w == ["h_ret->err"] for w in found), (name, found)
    end = text[text.index("int Ctx::end_call()"):]
    assert "h_ret->err" in end[:end.index("\n}")]
