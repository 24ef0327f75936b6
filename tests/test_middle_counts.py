"""GenTables::ev_mid, the evaluations of a middle instruction and the last one,
against their definition: every candidate of every mask for every pair of
registers that must still be read."""
import os
import subprocess

from pca_gb300.build import CSRC, LIBDIR, build_engine

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "gen_tables.h"
#include "pca_isa.h"
using namespace pcagb;

int main()
{
    const GenTables &t = gen_tables();
    if (t.ev_mid.size() != 2 * 128 * 64) return 1;
    /* evaluations of the last position after a write to r left mask m, of the
       classes that read x too (0: of all) */
    std::vector<uint32_t> last(128 * 64, 0);
    for (int m = 0; m < 128; m++)
        for (uint32_t r = 1; r < 8; r++)
            for (uint32_t e = t.pr_off[m * 8 + r]; e < t.pr_off[m * 8 + r + 1]; e++)
                for (uint32_t x = 0; x < 8; x++)
                    if (!x || (t.pr[e] & 7u) == x || (t.pr[e] >> 3 & 7u) == x)
                        last[(m * 8 + r) * 8 + x] += __builtin_popcount(t.pr[e] >> 6 & 0x3FFu);
    for (uint32_t d = 0; d < 2; d++)
        for (uint32_t m = 0; m < 128; m++)
            for (uint32_t A = 0; A < 8; A++)
                for (uint32_t B = 0; B < 8; B++) {
                    uint32_t want = 0;
                    for (uint32_t i = t.cand_off[m]; i < t.cand_off[m + 1]; i++) {
                        const uint32_t u = t.cand_uop[i], rd = UOP_RD(u);
                        if (d && t.cand_dupe[i]) continue;
                        const bool ua = A && UOP_A(u) != A && UOP_B(u) != A;   /* unread */
                        const bool ub = B && UOP_A(u) != B && UOP_B(u) != B;
                        if ((ua && ub) || (ua && rd == A) || (ub && rd == B)) continue;
                        want += last[((m | 1u << (rd - 1)) * 8 + rd) * 8 + (ua ? A : ub ? B : 0)];
                    }
                    const uint32_t got = t.ev_mid[((d * 128 + m) * 8 + A) * 8 + B];
                    if (got != want) {
                        printf("%u %u %u %u: %u, not %u\n", d, m, A, B, got, want);
                        return 1;
                    }
                }
    puts("ok");
    return 0;
}
"""


def test_middle_counts_are_their_definition(tmp_path):
    build_engine()
    src, exe = tmp_path / "mid.cpp", tmp_path / "mid"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, str(src),
                        os.path.join(LIBDIR, "libpcagb.so"), f"-Wl,-rpath,{LIBDIR}", "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
