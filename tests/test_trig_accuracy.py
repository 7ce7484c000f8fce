"""Host check that the table-driven sines and cosines (pagmo2_gb300/csrc/trig_table.h) are good to 2^-60, a quarter of
the last place of a sine of 2^-6 (tests/cpp/test_trig_table.cpp measures them)."""
from test_integer_arithmetic import build_and_run


def test_table_error(tmp_path):
    assert float(build_and_run(tmp_path, "test_trig_table")[1]) <= 2.0 ** -60
