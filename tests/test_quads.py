"""The quad arithmetic of the short-row CSR kernel, compiled for the host."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_whole_quads_up_to_the_largest_element_count(tmp_path):
    exe = tmp_path / "quads_check"
    subprocess.run(["g++", "-std=c++17", "-O1", str(HERE / "cpp" / "quads_check.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == "ok\n"
