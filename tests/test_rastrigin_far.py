"""Host check of rastrigin's squares outside the usual range (tests/cpp/test_rastrigin_far.cpp), built with g++."""
from test_integer_arithmetic import build_and_run


def test_rastrigin_far_squares(tmp_path):
    values, worst, violations = build_and_run(tmp_path, "test_rastrigin_far")
    assert int(values) == 800_000 and float(worst) <= 1.0 and int(violations) == 0
