"""Team shapes of plain solves, and the shared memory their blocks get, against
what the kernel lays out in it: host arithmetic, compiled with the host
compiler.  The kernel takes the team's kind from the launch: one block stages
in shared memory, as a cluster's blocks do, in front of its heap nodes; a ring's
blocks stage in global memory."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "team_shape.h"
using namespace gastar;
int main() {
    const uint32_t sms = 152;
    for (uint32_t kind = 0; kind < 4; ++kind)
        for (uint64_t cells : {100ull, 1ull << 17, (1ull << 17) + 1, 1ull << 24}) {
            if (kind != KIND_GRID && cells != 100) continue;
            for (uint32_t q : {0u, 1u, 33u, 512u, 513u, 4096u, 16384u, 65536u})
                for (uint32_t ew : {0u, 1u, 8u, 32u})
                    for (uint32_t w : {0u, 1u, 8u, 9u, 16u})
                        for (uint32_t cap : {0u, 1u, 2u, 16u, 17u, 200u})
                            for (int resident = 0; resident < 2; ++resident) {
                                gastar_config c;
                                std::memset(&c, 0, sizeof(c));
                                c.num_queues = q;
                                c.expansion_width = ew;
                                c.warps_per_block = w;
                                c.max_blocks = cap;
                                const PlainShape s = plain_shape(sms, kind, cells, c,
                                                                 [&](uint32_t, uint32_t, uint32_t) { return resident != 0; });
                                const uint32_t snodes = 20;
                                std::printf("%u %u %u %u %u %u %u %llu %d %d %zu %zu\n", kind, cap, w, ew, s.ew, s.ew_wide, s.W,
                                            (unsigned long long)s.blocks, (int)s.cluster, (int)s.ring(),
                                            block_smem_bytes(kind_bit(kind), s.W, s.ew_wide, s.ring(), snodes, false),
                                            block_smem_bytes(kind_bit(kind), s.W, s.ew_wide, s.ring(), snodes, true));
                            }
        }
}
"""


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    src, exe = d / "shape.cpp", d / "shape"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "cuda_a_star_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return [tuple(int(x) for x in line.split()) for line in out.splitlines()]


def test_blocks_lie_within_the_cap_and_the_kind_follows_them(shapes):
    assert any(s[9] for s in shapes) and any(s[8] for s in shapes)
    for kind, cap, w, fixed, ew, ew_wide, W, blocks, cluster, ring, _, _ in shapes:
        assert blocks >= 1 and 1 <= W <= 16 and 1 <= ew <= ew_wide <= 32
        assert not cap or blocks <= cap
        assert ring == (blocks > 1 and not cluster)
        assert not cluster or 2 <= blocks <= 16 and W <= 8
        # Puzzles with the automatic width widen on several blocks, clusters too.
        assert ew_wide == (min(32, 4 * ew) if blocks > 1 and kind < 3 and not fixed else ew)


def test_shared_memory_holds_what_the_kernel_lays_out(shapes):
    for kind, cap, w, fixed, ew, ew_wide, W, blocks, cluster, ring, heaps, buckets in shapes:
        entry, maxn = (32 if kind == 2 else 16), (8 if kind == 3 else 4)
        in_smem = blocks == 1 or cluster  # by the launch: team_ctas, cluster
        stage = 2 * W * max(ew, ew_wide) * maxn * entry if in_smem else 0
        nodes = W * 19 * 32 * entry  # 20 nodes: the partial buffer and 18 tree nodes, root included
        assert heaps >= stage + nodes
        assert buckets >= stage + nodes + W * 256
