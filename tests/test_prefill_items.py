"""Which kv head, tokens and position range a block of a prefill launch works on: the function that the kernel calls, compiled for
the host, over launches whose blocks can be listed and over ones whose items pass 2^32 / groups."""
import os
import subprocess

import q4gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(q4gpu.LIB_PATH)), "csrc")
PROGRAM = r"""
#include <stdio.h>
#include "q4_internal.h"
static int bad(const char *what, uint32_t g, uint32_t n_kvh, uint32_t whole, uint32_t ranges, uint64_t block) {
    printf("%s: %u groups x %u kv heads, %u whole, %u ranges, block %llu\n", what, g, n_kvh, whole, ranges, (unsigned long long)block);
    return 1;
}
int main() {
    const uint32_t groups[] = {1, 2, 3, 5, 37, 74, 148, 513, 23253, 23254, 23255, 33096, 46508, 65536, 65537, 1000003, 60000000};
    for (uint32_t g : groups)
        for (uint32_t n_kvh : {1u, 2u, 3u, 8u, 16u})
            for (uint32_t late : {0u, 1u, 7u, 68u, 147u})
                for (uint32_t ranges : {2u, 3u, 16u}) {
                    const uint64_t items = (uint64_t)g * n_kvh;
                    if (late >= items || items > 0x7fffffffull) continue;
                    const uint32_t whole = (uint32_t)(items - late);
                    const uint64_t blocks = whole + (uint64_t)late * ranges, step = blocks < 100000 ? 1 : g < 100000 ? 97 : 99991;
                    for (uint64_t b = 0; b < blocks; b = b + step < blocks || b + 1 >= blocks ? b + step : blocks - 1) {
                        for (uint64_t c = b < 3 ? 0 : b - 3; c <= b; c++) {
                            uint64_t item = c, range = 0;
                            if (c >= whole) { range = (c - whole) / late; item = whole + (c - whole) % late; }
                            const Q4PfItem r = q4i_pf_item((uint32_t)c, g, whole, late, ranges);
                            if (r.kh != item / g || r.group != item % g || r.range != range || r.ranges != (c >= whole ? ranges : 1u))
                                return bad("wrong item", g, n_kvh, whole, ranges, c);
                        }
                    }
                    for (uint32_t kh = 1; kh <= n_kvh; kh++) {   /* the last group of every kv head */
                        const uint64_t c = (uint64_t)kh * g - 1u;
                        if (c >= whole) continue;
                        const Q4PfItem r = q4i_pf_item((uint32_t)c, g, whole, late, ranges);
                        if (r.kh != kh - 1u || r.group != g - 1u) return bad("wrong last group", g, n_kvh, whole, ranges, c);
                    }
                }
    printf("ok\n");
    return 0;
}
"""


def test_items_of_a_launch(tmp_path):
    src, exe = tmp_path / "items.cpp", tmp_path / "items"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, "-I", "/usr/local/cuda/include", str(src), "-o", str(exe)],
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0, r.stdout
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
