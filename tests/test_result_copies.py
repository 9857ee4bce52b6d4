"""The ring that large results leave by: every byte in its place, whatever the sizes and the number of threads, and refusals in between
(host code, no GPU needed)."""
import subprocess
from pathlib import Path

PROBE = Path(__file__).with_name("result_copies_probe.cpp")


def test_results_arrive_whole_and_refusals_leave_nothing_behind(tmp_path):
    probe = tmp_path / "probe"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I/usr/local/cuda/include", str(PROBE), "-o", str(probe)], check=True)
    out = subprocess.run([str(probe)], check=True, capture_output=True, text=True, timeout=120).stdout
    assert out == "wrong 0 alive 0 waits 1\n"
