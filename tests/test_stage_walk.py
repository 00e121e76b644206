"""The walk of a persistent sweep CTA over its tiles (csrc/mgp_stage.cuh), compiled for
the host around a model of its mbarrier: a phase's wait returns at once when the barrier
stands in the other parity, as the hardware's does.  Copies that do not arrive within the
wait must end the walk without a store, and not before they have landed, whichever tile
they belong to."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mgpoisson2d_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "mgp_stage.cuh"
using namespace mgp;

// arguments: tiles, the tile whose copies are late (-1: none), polls until they land, polls a wait makes
int main(int, char** v) {
    const int n = atoi(v[1]), late = atoi(v[2]), delay = atoi(v[3]), limit = atoi(v[4]);
    int phases = 0, issued = 0, in_flight = 0, polls_left = 0, tile_no = 0, stored = 0, bad = 0;
    const auto issue = [&]() {
        in_flight = 1;
        polls_left = issued++ == late ? delay : 0;
    };
    const auto poll = [&](unsigned parity) {
        if (in_flight && polls_left-- <= 0) in_flight = 0, ++phases;
        return (phases & 1) != (int)parity;   // the phase of this parity is complete
    };
    const auto wait = [&](unsigned parity) {
        for (int k = 0; k < limit; ++k)
            if (poll(parity)) return true;
        return false;
    };
    issue();
    walk_tiles([&](int) {}, [&](unsigned parity) { if (!wait(parity)) bad = 1; },
               [&](int) {
                   if (bad) return TILE_LOST;
                   if (in_flight) exit(2);   // used before its copies had landed
                   const bool more = ++tile_no < n;
                   if (more) issue();
                   ++stored;
                   return more ? TILE_MORE : TILE_LAST;
               },
               [&](unsigned parity) { wait(parity); });
    printf("%d %d %d %d\n", stored, issued, in_flight, bad);
    return 0;
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("walk")
    (d / "walk.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, "-o", str(d / "walk"), str(d / "walk.cpp")], check=True)
    return lambda *a: [int(x) for x in
                       subprocess.run([str(d / "walk"), *map(str, a)], check=True, capture_output=True,
                                      text=True).stdout.split()]


@pytest.mark.parametrize("tiles", [1, 2, 3, 8])
def test_every_tile_is_stored_when_its_copies_arrive(walk, tiles):
    assert walk(tiles, -1, 0, 10) == [tiles, tiles, 0, 0]
    assert walk(tiles, tiles - 1, 7, 10) == [tiles, tiles, 0, 0]


@pytest.mark.parametrize("tiles,late", [(1, 0), (2, 0), (2, 1), (3, 1), (8, 7)])
def test_copies_that_are_late_land_before_the_walk_ends(walk, tiles, late):
    # later than one wait, within the second
    assert walk(tiles, late, 15, 10) == [late, late + 1, 0, 1]


def test_copies_that_never_arrive_end_the_walk(walk):
    stored, issued, in_flight, bad = walk(4, 2, 1000, 10)
    assert (stored, issued, in_flight, bad) == (2, 3, 1, 1)
