"""How the team CG shares the GPU's blocks among the systems of a batch (host code of pcg.cu, built here by itself): every system
gets a block, none more than it has shares, and no launch more than run together, on any number of SMs."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "sdot-ffi_b200", "csrc")
#: the clusters of 1, 2, 4, 8 and 16 blocks that run at once (of 148 SMs: a B200's answer)
CLUSTERS = {148: (148, 74, 33, 15, 7), 132: (132, 66, 30, 14, 6), 20: (20, 10, 4, 2, 1), 1: (1, 0, 0, 0, 0)}
MAIN = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <iostream>
#include "warp_on_host.h"
#include "internal.h"
namespace sdot {
#include "teams.inc"
}
using namespace sdot;
// in: SMs, the clusters of 1, 2, 4, 8 and 16 that run at once, the systems, their rows
// out: us an iteration, the bursts; a line per launch: problems, cluster size, then { problem, rank, size, team } a block
int main() {
    PcgDevice D;
    int np;
    std::cin >> D.blocks;
    for ( int &c : D.clusters ) std::cin >> c;
    std::cin >> np;
    std::vector<int> rows( np );
    for ( int &n : rows ) std::cin >> n;
    std::vector<PcgLaunch> launches;
    std::vector<int4> t;
    const double us = pcg_plan( rows, D, launches, t );
    std::printf( "%.1f %d %d %d\n", us, pcg_burst( us, true, false ), pcg_burst( us, false, false ), pcg_burst( us, false, true ) );
    for ( const PcgLaunch &l : launches ) {
        std::printf( "%d %d", l.nprob, l.cluster );
        for ( int k = l.block; k < l.block + l.nblock; ++k ) std::printf( " %d %d %d %d", t[ k ].x, t[ k ].y, t[ k ].z, t[ k ].w );
        std::printf( "\n" );
    }
}
"""


@pytest.fixture(scope="module")
def teams(tmp_path_factory):
    d = tmp_path_factory.mktemp("teams")
    src = open(os.path.join(CSRC, "pcg.cu")).read()

    def piece(a, b):
        i = src.index(a)
        return src[i:src.index(b, i)] + "\n"
    (d / "teams.inc").write_text(piece("constexpr int PCG_T", "\n") + piece("constexpr int PCG_W", "\n") +
                                 piece("// rows of a share", "struct Team") +
                                 piece("// the blocks of each of `np` problems", "cudaError_t launch_pcg"))
    (d / "main.cpp").write_text(MAIN)
    exe = str(d / "teams")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(d), "-I", HERE, "-I", CSRC, "-I", "/usr/local/cuda/include",
                    str(d / "main.cpp"), "-o", exe], check=True)

    def run(sms, rows):
        given = [sms, *CLUSTERS[sms], len(rows), *rows]
        out = subprocess.run([exe], input=" ".join(map(str, given)), check=True, capture_output=True, text=True).stdout
        us, *bursts = out.splitlines()[0].split()
        launches = []
        for line in out.splitlines()[1:]:
            nprob, cluster, *v = map(int, line.split())
            launches.append((nprob, cluster, list(zip(*[iter(v)] * 4))))
        return launches, float(us), [int(b) for b in bursts]
    return run


def shares(n):
    per = max(128, -(-(-(-n // 148)) // 32) * 32)
    return -(-n // per)


@pytest.mark.parametrize("sms", [148, 132, 20, 1])
@pytest.mark.parametrize("rows", [[9], [1000], [1000000], [500] * 8, [100003] * 9, [100003] * 17, [20011] * 65, [2001] * 150, [1000000] + [100] * 147,
                                  [1000000] + [3000] * 100, [4001, 100, 20011, 150]])
def test_every_system_has_its_blocks(teams, sms, rows):
    at = 0
    for nprob, cluster, blocks in teams(sms, rows)[0]:
        assert 1 <= nprob <= len(blocks) <= sms
        assert not cluster or nprob <= CLUSTERS[sms][cluster.bit_length() - 1]
        of = {}
        for problem, rank, size, team in blocks:
            assert team == problem and 0 <= rank < size
            of.setdefault(problem, []).append((rank, size))
        assert sorted(of) == list(range(nprob))
        for problem, team in of.items():
            assert [r for r, _ in team] == list(range(len(team))) and all(size == len(team) for _, size in team)
            # (a cluster's blocks past the shares do nothing)
            assert cluster in (0, len(team)) and (cluster or len(team) <= shares(rows[at + problem]))
        at += nprob
    assert at == len(rows)


@pytest.mark.parametrize("rows", [[100003] * 8, [100003] * 9, [100003] * 17, [50003] * 33, [20011] * 65, [20011] * 80, [20011] * 148])
def test_a_batch_of_large_systems_fills_the_sms(teams, rows):
    """the rows of the fullest block of each launch, together, against the rows an SM has to do at least: a third more at most (the
    clusters of one size left half of the SMs idle)"""
    at = fullest = 0
    for nprob, _, blocks in teams(148, rows)[0]:
        fullest += max(-(-rows[at + problem] // size) for problem, _, size, _ in blocks)
        at += nprob
    assert fullest <= 4 / 3 * sum(rows) / 148


@pytest.mark.parametrize("rows", [[1000], [20011], [100003], [1000000], [100003] * 9, [20011] * 65, [1000000] + [1000] * 7, [4000000]])
def test_a_launch_holds_the_stream_for_milliseconds(teams, rows):
    """10 ms where the solve is alone, 4 where others wait, and 8 iterations at least"""
    _, us, (alone, others, diagrams) = teams(148, rows)
    for burst, most, ms in ((alone, 256, 10), (others, 64, 4), (diagrams, 32, 4)):
        assert 8 <= burst <= most
        assert burst == 8 or burst * us <= 1000 * ms
        assert burst == most or (burst + 1) * us > 1000 * ms
