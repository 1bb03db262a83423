"""Who owns the memory of a launch, and until when (csrc/launch_slots.hpp), on a
model of streams, events, graphs and threads stepped in random order."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "thesis_gb300", "csrc")


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("slots") / "model")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, os.path.join(HERE, "launch_slots_model.cpp"),
                    "-o", exe, "-lpthread"], check=True, timeout=300)
    return exe


def test_no_launch_loses_its_memory(model):
    for seed in range(400):
        r = subprocess.run([model, "slots", str(seed), "3000"], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, (seed, r.returncode, r.stdout)


def test_slots_taken_in_turn_are_caught(model):
    """Four buffers in turn, remade when a larger one is wanted: each of the
    ways in which a launch loses its memory shows."""
    seen = set()
    for seed in range(200):
        r = subprocess.run([model, "ring", str(seed), "3000"], capture_output=True, text=True, timeout=60)
        if r.returncode:
            seen.add(r.stdout.split(": ")[1].strip())
    assert "memory of a running launch cleared" in seen
    assert "freed memory cleared" in seen
