"""The row_ptr arithmetic of the triplet converter, compiled for the host."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_rows_starting_at_up_to_the_largest_row_count(tmp_path):
    exe = tmp_path / "row_span_check"
    subprocess.run(["g++", "-std=c++17", "-O1", str(HERE / "cpp" / "row_span_check.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == "ok\n"
