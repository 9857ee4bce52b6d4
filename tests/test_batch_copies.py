"""The stream and events that tg_batch's results leave by: a failure half way leaves nothing behind (host code, no GPU needed)."""
import subprocess
from pathlib import Path

PROBE = Path(__file__).with_name("batch_copies_probe.cpp")


def test_a_failed_set_up_leaves_nothing_behind(tmp_path):
    probe = tmp_path / "probe"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include", str(PROBE), "-o", str(probe)], check=True)
    out = subprocess.run([str(probe)], check=True, capture_output=True, text=True).stdout
    # layers of 197120 parameters: three of them exceed 2^19 (the first with 256 of the final norm)
    assert out == "6:1215488 3:624128 0:32768 wrong 0 alive 0\n"
