"""Host check of the table-driven cosine at and next to whole turns (tests/cpp/test_trig_turns.cpp), built with g++."""
from test_integer_arithmetic import build_and_run


def test_cosine_never_exceeds_one(tmp_path):
    values, rows, violations = build_and_run(tmp_path, "test_trig_turns")
    assert int(values) > 4_000_000 and int(rows) > 1000 and int(violations) == 0
