"""No vote or reduction of the search kernel has an operand that is a constant
in any instantiation.

A vote on a compile-time constant in the grid kernel (a flag that only hash
tables can raise) hung every warp on the GPU, all lanes in straight code between
the expansion loop and the block barrier; one reduction of a run-time word in
its place ran.  The host compiler, after inlining every instantiation, refuses
an operand that it knows."""
import os
import subprocess

import pytest

import kernel_host

MAIN = r"""
#include "votes.h"
#include "plugin.cuh"
namespace gastar {
template <int BYTES> struct State { unsigned char b[BYTES]; };
template <int BYTES> void gen(const State<BYTES>& a, State<BYTES>& o, bool& ex, uint32_t& cost, unsigned char i) {
    o = a;
    o.b[0] += i;
    ex = o.b[0] != 0;
    cost = 1 + i;
}
template <int BYTES> uint32_t heur(const State<BYTES>& s) { return s.b[0]; }
#define TEAMS(T, ...)                                                               \
    template void run_instance<__VA_ARGS__, T, TEAM_BLOCK>(const LaunchParams&, const TeamRef); \
    template void run_instance<__VA_ARGS__, T, TEAM_RING>(const LaunchParams&, const TeamRef);  \
    template void run_instance<__VA_ARGS__, T, TEAM_CLUSTER>(const LaunchParams&, const TeamRef);
#define DOM(...) TEAMS(256, __VA_ARGS__) TEAMS(512, __VA_ARGS__)
#if PART == 0
DOM(SlidingDom<3>) DOM(SlidingDom<4>)
#elif PART == 1
DOM(SlidingDom<5>) DOM(GridDom)
#elif PART == 2
TEAMS(256, PluginDom<State<8>, 4, gen<8>, heur<8>>) TEAMS(256, PluginDom<State<20>, 33, gen<20>, heur<20>>)
TEAMS(256, PluginDom<State<32>, 1, gen<32>, heur<32>>)
#endif
}
"""


def _compile(dst, part):
    src = os.path.join(dst, "main%d.cpp" % part)
    with open(src, "w") as f:
        f.write(MAIN)
    return subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-DPART=%d" % part, "-c", src, "-o", src + ".o"],
                          capture_output=True, text=True)


@pytest.mark.parametrize("part", [0, 1, 2])
def test_no_operand_folds_to_a_constant(tmp_path, part):
    kernel_host.rewrite(str(tmp_path), "votes.h")
    r = _compile(str(tmp_path), part)
    assert r.returncode == 0, r.stderr[:3000]


def test_a_vote_per_flag_is_refused(tmp_path):
    """The form that hung: bit 0 is raised by hash tables only."""
    one = "            flags = uniform(flags);\n"
    each = ("            flags = (__any_sync(kFull, (flags & 1u) != 0) ? 1u : 0u) |\n"
            "                    (__any_sync(kFull, (flags & 2u) != 0) ? 2u : 0u);\n")

    def plant(name, text):
        if name == "search.cuh":
            assert text.count(one) == 1
            text = text.replace(one, each)
        return text

    kernel_host.rewrite(str(tmp_path), "votes.h", plant)
    assert _compile(str(tmp_path), 0).returncode == 0  # puzzles raise both
    r = _compile(str(tmp_path), 1)
    assert r.returncode != 0 and "a vote or reduction of a constant" in r.stderr and "GridDom" in r.stderr
