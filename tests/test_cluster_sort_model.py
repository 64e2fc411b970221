"""The exchanges of the cluster sort (k_codes_sort) under any delay of its
messages: an exhaustive search over the schedules of three blocks, with the
barriers that the kernel takes (cluster_exchange.h, compiled by the model too).

The pairs of a pass go where their digits say: from every block to every block;
from each block to itself alone (a digit that all nodes of a block's range
share: coincident nodes, or one far outlier); from each to the next; between two
blocks with the third empty."""
import itertools
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
FLOWS = {"all": "111111111", "own": "100010001", "next": "010001100", "empty": "110110000"}


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "a C++ compiler is required"
    out = {}
    for bars in (None, 1):
        exe = str(tmp_path_factory.mktemp("model") / "model")
        subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe] +
                       ([f"-DCS_COUNT_BARS={bars}"] if bars else []) +
                       [os.path.join(HERE, "cluster_sort_model.cpp")], check=True)
        out[bars] = exe

    def run(bars, passes):
        return subprocess.run([out[bars], "3", "".join(FLOWS[p] for p in passes)], check=True,
                              capture_output=True, text=True, timeout=300).stdout.strip()
    return run


@pytest.mark.parametrize("passes", list(itertools.product(("all", "own", "next"), repeat=3)),
                         ids="-".join)
def test_no_schedule_reads_another_pass(model, passes):
    assert model(None, passes).startswith("ok ")


def test_no_schedule_with_an_empty_block_reads_another_pass(model):
    assert model(None, ("empty",) * 3).startswith("ok ")


def test_the_model_finds_the_race_of_a_single_barrier(model):
    assert model(1, ("own",) * 3) == "wrong: counts read"
    assert model(1, ("empty",) * 3) == "wrong: counts read"
    assert model(1, ("all",) * 3).startswith("ok ")
