"""The launch shape of the trainers that hold one or two walks to a warp (dg_pair_grid.h), for
every worker bound: as many walks under way as asked for, rounded up to whole blocks as the
other trainers' launches round, and no more than the GPU holds."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gdistger-re_b200", "csrc")
PROGRAM = """
#include "dg_pair_grid.h"
#include <cstdio>
#include <cstdlib>
int main(int, char **v) {
    const dgs::PairGrid most{atoi(v[1]), atoi(v[2]), (uint32_t)atoi(v[3])};
    for (uint32_t want = 0; want <= 5000; want++) {
        const dgs::PairGrid g = dgs::pair_grid(want, most);
        printf("%d %d %u\\n", g.blocks, g.warps, g.walks);
    }
    const dgs::PairGrid g = dgs::pair_grid(~0u, most);
    printf("%d %d %u\\n", g.blocks, g.warps, g.walks);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("grid")
    (d / "grid.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(d / "grid.cpp"), "-o", str(d / "grid")], check=True)
    return str(d / "grid")


@pytest.mark.parametrize("blocks,warps,walks", [(296, 8, 2), (148, 8, 1), (148, 8, 2), (1, 8, 2)])
def test_every_worker_bound(program, blocks, warps, walks):
    out = subprocess.run([program, str(blocks), str(warps), str(walks)], check=True, capture_output=True, text=True).stdout
    shapes = [tuple(map(int, line.split())) for line in out.splitlines()]
    full = blocks * warps * walks
    assert shapes[0] == shapes[-1] == (blocks, warps, walks)
    for want, (b, w, k) in enumerate(shapes[:-1]):
        if want == 0:
            continue
        assert 1 <= b <= blocks and 1 <= w <= warps and 1 <= k <= walks
        under_way = b * w * k
        assert under_way >= min(want, full)
        assert under_way == want if want < warps else under_way < want + w * k or b == blocks and k == 1
