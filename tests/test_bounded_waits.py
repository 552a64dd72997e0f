"""The bounded wait for bulk copies into shared memory, compiled for the host with a barrier that
completes at a given poll.

A wait that runs out reports it, and gives the copies as long again: one that is still in flight when
its block ends would land in the memory of the block that comes after it."""
import os
import re
import subprocess

from tests.test_launch_order import CSRC

HOST = r"""
#include <cstdio>
#include <cstdlib>
#define __device__
#define __forceinline__ inline
static long polls, lands;
static bool mbar_test(unsigned long long *, unsigned) { return polls++ >= lands; }
static void __nanosleep(unsigned) {}
%s
int main(int, char **v)
{
    lands = atol(v[1]);
    const bool ok = mbar_wait(nullptr, 0);
    printf("%%d %%ld\n", (int)ok, polls);
}
"""


def test_limits(tmp_path):
    src = open(os.path.join(CSRC, "msod_device.cuh")).read()
    fn = re.search(r"__device__ __forceinline__ bool mbar_wait\(.*?\n\}\n", src, re.S).group(0)
    cpp, exe = tmp_path / "wait.cpp", tmp_path / "wait"
    cpp.write_text(HOST % fn)
    subprocess.run(["g++", "-O1", "-o", str(exe), str(cpp)], check=True)

    def run(lands):
        ok, polls = subprocess.run([str(exe), str(lands)], capture_output=True, text=True, check=True).stdout.split()
        return ok == "1", int(polls)

    limit = 1 << 20
    assert run(0) == (True, 1)
    assert run(limit - 1) == (True, limit)
    assert run(limit) == (False, limit + 1)  # late: reported, and waited for
    assert run(2 * limit - 1) == (False, 2 * limit)
    assert run(10 * limit) == (False, 2 * limit)  # never: still bounded
