"""What may stand ahead of a kernel that starts early (CPU check of the launch code).

launch_after lets a kernel start before the operation ahead of it on the stream has finished; the
kernel waits (griddepcontrol.wait) only before its first reduction, so everything it reads until then
has to be complete before that operation starts.  A copy queued by the same function -- the
derivative matrices on their way to the constant bank, which a kernel reads from its first pass on -- is
not: a function that copies or clears device memory launches its kernel the ordinary way.
"""
import os
import re

import pytest

from tests.test_noalloc_source import code_only

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "minisod2d_gb300", "csrc")
QUEUED = re.compile(r"\bcuda(Memcpy\w*|Memset\w*)\s*\(")
FUNCTION = re.compile(r"^\{\n(.*?)^\}", re.M | re.S)


def _block_end(code, at):
    """End of the innermost { } block that holds position `at`."""
    depth = 0
    for i in range(at, len(code)):
        depth += {"{": 1, "}": -1}.get(code[i], 0)
        if depth < 0:
            return i
    return len(code)


def _faults(code):
    """Copies that a launch_after of the same function follows (no block on the way returns first)."""
    out = []
    for body in FUNCTION.findall(code):
        for m in QUEUED.finditer(body):
            end = _block_end(body, m.start())
            while end < len(body) and not re.search(r"[;{}]\s*return\s[^;]*;\s*$", body[m.start():end]):
                end = _block_end(body, end + 1)
            if "launch_after" in body[m.start():end]:
                out.append(m.group(0))
    return out


def test_finder():
    bad = "int f()\n{\n if (c) { cudaMemcpyToSymbolAsync(a, b); if (e) return e; }\n return launch_after(k, 1);\n}\n"
    assert len(_faults(bad)) == 1
    assert not _faults(bad.replace("return e; }", "return e; k<<<1, 2>>>(); return 0; }"))


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))))
def test_no_copy_ahead_of_an_early_start(name):
    assert not _faults(code_only(open(os.path.join(CSRC, name)).read())), name


def test_matrices_ahead_of_the_zeroing():
    code = code_only(open(os.path.join(CSRC, "msod_capi.cu")).read())
    calls = [b for b in FUNCTION.findall(code) if "launch_diffu_plain" in b]
    assert calls
    for body in calls:
        prepare = body.index("prepare_diffu_plain")
        zero = re.search(r"\b(launch_zero|zero_outputs)\(", body).start()
        assert prepare < zero < body.index("launch_diffu_plain")
