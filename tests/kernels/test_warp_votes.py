"""A warp whose lanes each keep what they do next has to find one answer wherever the way forks: a test that does not wait has to be a vote of the whole
warp (over __activemask() it is one of the lanes that happen to be there), in a role whose lanes cannot have left each other. Read from the sources."""

import re

from nanonemo_b200.csrc import build


def _code(name):
    return re.sub(r"//[^\n]*", "", (build.HERE / name).read_text())


def _mma_role(name, end):
    text = (build.HERE / name).read_text()
    start = text.index("MMA issuer (warp-uniform")
    return re.sub(r"//[^\n]*", "", text[start:text.index(end, start)])


def test_no_vote_is_taken_over_the_lanes_that_happen_to_be_there():
    names = [p.name for ext in ("*.cu", "*.cuh", "*.inc") for p in build.HERE.glob(ext)]
    assert names and not [n for n in names if "__activemask" in _code(n)]
    header = _code("sm100.cuh")
    for function in ("mbar_test_warp", "mbar_wait_warp"):
        body = header[header.index(f"bool {function}("):]
        assert "return __all_sync(0xffffffffu, " in body[:body.index("\n}")]


def test_attention_backward_waits_as_a_warp_where_it_also_tests():
    role = _mma_role("flash_bwd.cu", "if (warp == 2")
    assert "mbar_test_warp(" in role and not re.findall(r"mbar_wait\(", role)
    for m in re.finditer(r"next_known\(", role):
        assert role[:m.start()].endswith("__all_sync(0xffffffffu, ")


def test_attention_forward_does_not_test():
    """Its lanes wait for themselves, so nothing may depend on when they ask, and each lets go of the answer that it has read."""
    role = _mma_role("flash_fwd.cu", "\n  } else {")
    assert "mbar_wait(" in role and not re.findall(r"test|_sync\(|\blane\b(?! == 0\) fail_role)", role)
    assert re.search(r"^ *mbar_arrive\(bar_ne", role, re.M)
    assert "kNextReaders = 32 + 4;" in _code("flash_fwd.cu")
