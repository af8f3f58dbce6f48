"""The split plan of packed attention at sizes that no cache holds: `tests/attention_plan_walk.cpp` walks through the
pieces of random and extreme calls on the host, with the header the kernel and its launcher are built from."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_unit_is_in_one_piece_with_a_slot_and_a_chunk(tmp_path):
    binary = str(tmp_path / "attention_plan_walk")
    build = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I",
                            os.path.join(ROOT, "qwencore_b200", "csrc", "kernels"),
                            os.path.join(ROOT, "tests", "attention_plan_walk.cpp"), "-o", binary],
                           capture_output=True, text=True)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([binary], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout[-1000:]
    counts = dict(part.split("=") for part in run.stdout.split()[1:])
    assert 0 < int(counts["wide"]) < int(counts["dynamic"]) < int(counts["calls"])
