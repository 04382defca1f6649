"""The stage ring that two consumer groups of the one-column kernel share (csrc/ring.h), modelled on the CPU: no wait may pass before its
stage has landed, and no barrier may be armed while it is pending, whatever the order in which loads land."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fast-llm_b200", "csrc")


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("ring") / "ring_model")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, os.path.join(HERE, "ring_model.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("seed", range(4))
def test_slots_of_a_group_are_its_own(model, seed):
    r = subprocess.run([model, str(seed), "4000"], stdout=subprocess.PIPE, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


def test_the_model_finds_what_slots_passed_on_do(model):
    r = subprocess.run([model, "1", "4000", "shared"], stdout=subprocess.PIPE, text=True, timeout=300)
    assert r.returncode == 1 and "before its stage had landed" in r.stdout
