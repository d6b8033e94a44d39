"""The key-row streams (csrc/key_stream.cuh) on a host model of the barriers,
with one row's copy that never lands (or none): the stream ends by itself,
arms no slot whose copy is out, and waits for what it has issued.  CPU only."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fpga-tfhe_gb300", "csrc")


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("streams") / "key_streams")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", exe, os.path.join(HERE, "key_streams.cpp")],
                   check=True, capture_output=True)

    def run(what, lost):
        return subprocess.run([exe, what, str(lost)], capture_output=True, text=True, timeout=60).stdout.split("\n")[:-1]

    return run


# no row lost; the first, one whose slot has a next use, the last two
@pytest.mark.parametrize("stream,rows", [("products2", 12), ("products3", 18)])
def test_product_stream_ends_by_itself(model, stream, rows):
    for lost in (-1, 0, 3, 6, rows - 2, rows - 1):
        assert model(stream, lost) == [], lost


# rows only of the items that rotate: zeros first, last, in a row; none; no items
@pytest.mark.parametrize("stream,rows", [("rotations2", [4, 7, 16, 18, 22, 23]), ("rotations3", [0, 3, 12, 16, 17]),
                                         ("no_rotation", []), ("no_items", [])])
def test_product_stream_copies_what_is_used(model, stream, rows):
    for lost in [-1] + rows:
        assert model(stream, lost) == [], lost


# shared rings: streamed in line, by a producer warp, for lane pairs, for two halves
@pytest.mark.parametrize("stream", ["ring", "producer_warp", "lane_pairs", "pair"])
def test_ring_ends_by_itself(model, stream):
    for lost in (-1, 0, 2, 4, 9, 13, 16, 17):
        assert model(stream, lost) == [], lost
