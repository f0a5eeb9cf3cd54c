"""A team's list of candidates packs a slot and its row into 32 bits: teams are
used only where every slot of the launch fits (pbf_kernels.h, pbf_team.cuh)."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mtlphys_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include "pbf_kernels.h"
using namespace mpb;
int main() {
    for (unsigned n : {1u, 300u, 16384u, 16385u, 1u << 28})
        for (unsigned end : {n, 20000u, kTeamMaxSlots - 1u, kTeamMaxSlots, kTeamMaxSlots + 1u, 1u << 29, 1u << 30})
            if (end >= n) std::printf("%u %u %u\n", n, end, team_lanes(n, end));
}
"""


def test_teams_only_where_their_slots_fit(tmp_path):
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", "/usr/local/cuda/include", "t.cpp", "-o", "t"],
                   cwd=tmp_path, check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout
    lines = [tuple(map(int, x.split())) for x in out.splitlines()]
    assert any(lanes for _, _, lanes in lines) and any(end > 1 << 28 for _, end, _ in lines)
    for n, end, lanes in lines:
        fits = all(((end - 1) | y << 28 | z << 30) & 0x0FFFFFFF == end - 1 for y in range(3) for z in range(3))
        assert lanes == (16 if n <= 16384 and fits else 0), (n, end)
