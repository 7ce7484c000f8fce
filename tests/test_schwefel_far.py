"""Host check of schwefel's elements outside the usual range (tests/cpp/test_schwefel_far.cpp), built with g++."""
from test_integer_arithmetic import build_and_run


def test_schwefel_far_elements(tmp_path):
    values, small, large, violations = build_and_run(tmp_path, "test_schwefel_far")
    assert int(values) > 400_000 and int(violations) == 0
    assert float(small) <= 1.5 and float(large) <= 1.0
