"""Host check of DTLZ's fixed-point squares (tests/cpp/test_unit_square.cpp), built with g++."""
from test_integer_arithmetic import build_and_run


def test_centred_squares(tmp_path):
    values, worst, mean, violations = build_and_run(tmp_path, "test_unit_square")
    assert int(values) > 390_000 and int(violations) == 0
