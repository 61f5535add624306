"""The decode attention's ring of stages (csrc/dec_ring.h) on a CPU: a C++ driver (tests/dec_ring_order.cpp, compiled here with g++) plays the
warps of a block through it in random orders, with copies that land at random times."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def play(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("ring") / "dec_ring_order")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "qwenny_b200", "csrc"),
                    os.path.join(ROOT, "tests", "dec_ring_order.cpp"), "-o", exe], check=True)
    return lambda look: [int(x) for x in subprocess.run([exe, str(look)], check=True, capture_output=True, text=True).stdout.split()]


def test_quads_read_their_own_stages_whatever_the_order(play):
    """Two and four quads, a split per block and runs of one to six splits of 1 to 22 stages: every stage is read when it is there and before
    another takes its place, no slot is armed twice, nothing is copied into the merge's slots, and nobody waits for ever."""
    assert play(1) == [0] * 5


def test_a_parity_alone_lets_a_quad_read_too_early(play):
    """Without the look at the slot's number a quad that comes to a slot whose last stage, another quad's, has not landed is let through: the
    driver sees it in each of the five forms."""
    assert all(n > 0 for n in play(0))
