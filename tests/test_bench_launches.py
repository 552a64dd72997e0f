"""bench.py's kernel count per step: the line above which the diffusion prepares a constant bank is the
library's (CPU check against its source)."""
import os
import re

import bench

SRC = os.path.join(bench.ROOT, "minisod2d_gb300", "csrc", "msod_diffu.cu")


def _source_line(P):
    expr = re.search(r"diffu_const_points\(\)\s*\{\s*return ([^;]+);", open(SRC).read()).group(1)
    py = re.sub(r"(.+?) \? (.+?) : \((.+?) \? (.+?) : (.+?)\)$", r"(\2) if (\1) else ((\4) if (\3) else (\5))", expr)
    return eval(py.replace("||", "or"), {"P": P})


def test_launches_per_step():
    for P in range(1, 9):
        line = _source_line(P)
        assert bench.launches_per_step(P, line) == 5 and bench.launches_per_step(P, line - 1) == 4
    assert bench.launches_per_step(4, 64 ** 3 * 125) == 5  # plain_64
    assert bench.launches_per_step(4, 32 ** 3 * 125) == 4  # plain_32
