"""Host check of griewank's factors next to 0 (tests/cpp/test_trig_small.cpp), built with g++."""
from test_integer_arithmetic import build_and_run


def test_griewank_small_factors(tmp_path):
    values, worst, worst_product, violations = build_and_run(tmp_path, "test_trig_small")
    assert int(values) > 500_000 and int(violations) == 0
    assert float(worst) <= 2.0 and float(worst_product) <= 1.0
