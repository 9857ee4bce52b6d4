"""The ring that large results leave by: every byte in its place, whatever the sizes and the number of threads, and refusals in between
(host code, no GPU needed)."""
import os
import subprocess
from pathlib import Path

import pytest

PROBE = Path(__file__).with_name("result_copies_probe.cpp")


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    program = tmp_path_factory.mktemp("ring") / "probe"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I/usr/local/cuda/include", str(PROBE), "-o", str(program)], check=True)
    return program


def test_results_arrive_whole_and_refusals_leave_nothing_behind(probe):
    out = subprocess.run([str(probe)], check=True, capture_output=True, text=True, timeout=120).stdout
    assert out == "wrong 0 alive 0 waits 1\n"


def test_processors_are_those_the_caller_may_run_on(probe):
    mine = sorted(os.sched_getaffinity(0))
    for allowed in {1, len(mine)}:
        out = subprocess.run([str(probe), "processors"], check=True, capture_output=True, text=True, timeout=120,
                             preexec_fn=lambda: os.sched_setaffinity(0, mine[:allowed])).stdout
        assert int(out) == allowed
