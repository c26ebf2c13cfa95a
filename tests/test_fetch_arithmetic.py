"""The dynamic ray fetch's index arithmetic (csrc/cpt_fetch.h), compiled as host C++ and run over small
and the largest queries: every item once, nothing past the end, and a positive number of lanes.  (A
query of 2^31 - 2 rays is 100 GB; the kernel itself is not run at that size.)"""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cudapathtracing_gb300", "csrc")

PROGRAM = r"""
#include "cpt_fetch.h"
#include <cstdio>
#include <algorithm>
using namespace cpt;
// One query: `warps` warps in turn fetch 32 items each from the counter at `start` until they have
// seen the end.  Returns the items handed out, or -1 after a wrong one.
static long long run(int n, int warps, uint32_t start)
{
    uint32_t counter = start;
    long long items = 0;
    for (int w = 0; w < warps; ++w)
        for (bool ended = false; !ended;) {
            const uint32_t base = counter;
            counter += 32;
            ended = fetch_ends(base, 32, n);
            for (int k = 0; k < 32; ++k) {
                const uint32_t r = base + (uint32_t)k;
                if (is_item(r, n)) {
                    if ((int)r < 0) return -1;
                    ++items;
                } else if (!ended) return -1;
            }
        }
    return items;
}
int main()
{
    const int top = 0x7ffffffe;
    for (int n : {1, 2, 31, 32, 33, 1000, top - 40000, top - 1, top}) {
        const uint32_t start = n > 4096 ? (uint32_t)n - 4096u : 0u;
        for (int warps : {1, 7, 5472, 20000})
            if (run(n, warps, start) != (long long)n - start) return std::printf("items n=%d warps=%d\n", n, warps), 1;
        for (int warps : {1, 7, 5472, 20000}) {
            const int lanes = spread_lanes(n, warps);
            const long long want = std::min(32LL, ((long long)n + warps - 1) / warps);
            if (lanes != want) return std::printf("lanes n=%d warps=%d: %d\n", n, warps, lanes), 1;
        }
    }
    return 0;
}
"""


def test_every_item_once_up_to_the_largest_query(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "fetch.cpp", tmp_path / "fetch"
    src.write_text(PROGRAM)
    subprocess.check_call([gxx, "-std=c++17", "-O1", "-fwrapv", "-I" + CSRC, str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
