"""Room for the on-chip solvers' launches (resident_room.h), on the CPU.

The blocks of a grouped launch wait for one another.  Whatever launches come,
and in whatever order they end, a grouped launch and all that may run beside it
must not be able to touch more SMs than there are; and nothing waits that need
not."""
import os
import random
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 148

MAIN = r"""
#include <cstdio>
#include "resident_room.h"
using namespace sedi;
// Lines: "blocks group n (blocks group)*n" -> held grouped, then the n waits.
int main() {
	int blocks, group, n;
	while (scanf("%d %d %d", &blocks, &group, &n) == 3) {
		std::vector<RoomUse> run;
		for (int i = 0; i < n; i++) {
			int b, g;
			if (scanf("%d %d", &b, &g) != 2) return 1;
			run.push_back(room_use(b, g, 148));
		}
		const RoomUse u = room_use(blocks, group, 148);
		printf("%d %d", u.held, (int)u.grouped);
		for (char w : room_waits(run, u, 148)) printf(" %d", (int)w);
		printf("\n");
	}
}
"""


@pytest.fixture(scope="module")
def waits(tmp_path_factory):
    d = tmp_path_factory.mktemp("room")
    (d / "main.cc").write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I",
                           os.path.join(REPO, "sedi_b200", "csrc"), str(d / "main.cc"), "-o", str(d / "room")])

    def call(new, running):
        line = " ".join(str(v) for v in (*new, len(running), *(v for r in running for v in r)))
        out = subprocess.run([str(d / "room")], input=line + "\n", capture_output=True, text=True, check=True).stdout
        return [int(v) for v in out.split()]
    return call


def test_a_two_per_sm_launch_may_touch_every_sm(waits):
    # 256 blocks, two of which fit an SM, and 20 that need an SM each.
    assert waits((20, 20), [(256, 32)]) == [20, 1, 1]
    assert waits((256, 32), [(20, 20)]) == [148, 1, 1]


def test_single_block_launches_count(waits):
    assert waits((144, 144), [(148, 1)]) == [144, 1, 1]   # a grouped one waits for them
    assert waits((148, 1), [(144, 144)]) == [148, 0, 1]   # and they for it
    assert waits((148, 1), [(148, 1), (30, 1)]) == [148, 0, 0, 0]  # among themselves nothing


def test_launches_that_fit_run_side_by_side(waits):
    assert waits((64, 64), [(64, 64)]) == [64, 1, 0]
    assert waits((20, 20), [(64, 64), (64, 64)]) == [20, 1, 0, 0]
    assert waits((21, 21), [(64, 64), (64, 64)]) == [21, 1, 1, 0]  # the oldest
    assert waits((40, 1), [(100, 1), (60, 60)]) == [40, 0, 0, 1]   # a single one only for the grouped


def test_random_launch_orders_leave_room(waits):
    """Launches come and end at random (one ends only when those it waits for
    have); those of which none starts behind another, directly or through
    others, may run at once."""
    rng = random.Random(5)

    def apart(i, j):  # one starts behind the other
        return i in after[j] or j in after[i]

    def most(g):  # SMs of g and launches that may all run at once with it
        def grow(total, rest):
            return max([total] + [grow(total + min(shape[i][0], SMS), [j for j in rest[k + 1:] if not apart(i, j)])
                                  for k, i in enumerate(rest)])
        return grow(min(shape[g][0], SMS), [i for i in live if i != g and not apart(i, g)])

    for _ in range(40):
        live, after = [], {}  # ids oldest first; after[i]: launches i starts behind
        shape = {}
        for k in range(14):
            group = rng.choice([1, 1, rng.randint(2, 148)])
            blocks = min(group * rng.randint(1, 40), 296 if rng.random() < 0.3 else 148) // group * group or group
            got = waits((blocks, group), [shape[i] for i in live])
            shape[k] = (blocks, group)
            after[k] = set()
            for i, w in zip(live, got[2:]):
                if w:
                    after[k] |= {i} | after[i]
            live.append(k)
            for g in live:
                if shape[g][1] > 1:
                    assert most(g) <= SMS
            ready = [i for i in live if not after[i] & set(live)]
            for i in ready:
                if rng.random() < 0.35:
                    live.remove(i)
