"""Fork and join of work on a side stream (csrc/side_stream.h) on recorded CUDA
calls: a call that fails in between still makes the caller's stream wait for what
it launched on the side stream."""

from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
FORK = "record main r;wait side r;launch side;"
JOIN = "record side d;wait main d;"


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = tmp_path_factory.mktemp("side") / "side_work"
    subprocess.run(["g++", "-std=c++17", "-I/usr/local/cuda/include",
                    f"-I{ROOT / 'aospectrum_b200' / 'csrc'}", str(ROOT / "tests/side_work_main.cpp"),
                    "-o", str(out)], check=True, capture_output=True)
    return out


@pytest.mark.parametrize("steps,fail_at", [(0, -1), (1, -1), (3, -1), (1, 0), (3, 2)])
def test_every_fork_is_joined(program, steps, fail_at):
    got = subprocess.run([str(program), str(steps), str(fail_at)], check=True, capture_output=True,
                         text=True).stdout.split(" ", 2)
    done = steps if fail_at < 0 else fail_at + 1
    assert got[0] == ("0" if fail_at < 0 else "7")
    assert got[1] == "0"   # events destroyed
    assert got[2].strip() == (FORK + JOIN) * done
