"""Host check of the short table cosine of the ackley, ZDT4 and DTLZ rows (tests/cpp/test_cos_short.cpp), built with
g++."""
from test_integer_arithmetic import build_and_run


def test_short_cosine(tmp_path):
    values, worst, violations = build_and_run(tmp_path, "test_cos_short")
    assert int(values) > 2_000_000 and int(violations) == 0 and float(worst) <= 2.0 ** -57
