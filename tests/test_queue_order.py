"""The tile queue of light manifold rounds (csrc/extremz_queue.h, compiled here
for the host) on a model of relaxed memory: every entry is taken and no block waits
in vain.  With the count of finished entries read without acquire order, a block can
leave with the ticket of an entry pushed later; the last block to push then waits
for that entry until its limit and asks for the dense pass (the labels stay right,
the search has cost a stall)."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "extrem_z_b200", "csrc")


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("queue") / "queue_model")
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", CSRC,
                    os.path.join(HERE, "native", "queue_model.cpp"), "-o", exe], check=True)
    return lambda order, seeds: [int(x) for x in subprocess.run(
        [exe, order, str(seeds)], check=True, capture_output=True, text=True,
        timeout=300).stdout.split()[1::2]]


def test_every_entry_is_taken(model):
    assert model("acquire", 5000) == [0, 0]


def test_without_the_order_blocks_wait_in_vain(model):
    left, waited = model("relaxed", 300)
    assert left == 0 and waited > 0
