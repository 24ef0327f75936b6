"""The value forms of the last positions (csrc/value_forms.h), on the host:
the closed-form keys of a target against evaluating every form, on edge and
random words; and the forms against the generator, for all 128 liveness
masks: every value class is exactly one form's, but for the copies of a
register and the zeros that no solving program needs, and every last
instruction a form names is in the operand-pair list it is looked up in."""
import os
import subprocess

from pca_gb300.build import CSRC, LIBDIR, build_engine

PROGRAM = r"""
#include <cstdio>
#include <map>
#include <random>
#include <set>
#include <vector>
#include "value_forms.h"
#include "gen_tables.h"
using namespace pcagb;

static int fail(const char *what, unsigned a, unsigned b, unsigned c, unsigned d)
{
    printf("%s: %x %x %x %x\n", what, a, b, c, d);
    return 1;
}

/* values on two tests to a word: (v, x, t) and (w, y, s) */
static int keys(uint32_t v, uint32_t x, uint32_t t, uint32_t w, uint32_t y, uint32_t s)
{
    const uint32_t V = v | w << 16, X = x | y << 16, G = t | s << 16;
    for (uint32_t f = 0; f < kPairForms; f++)
        if (pair_value2(f, V, X) != (pair_value(f, v, x) | pair_value(f, w, y) << 16))
            return fail("pair_value2", f, V, X, 0);
    for (uint32_t f = 0; f < kSelfForms; f++)
        if (self_value2(f, V) != (self_value(f, v) | self_value(f, w) << 16))
            return fail("self_value2", f, V, 0, 0);
    if (pair_mask2(V, X, G) != (pair_mask(v, x, t) & pair_mask(w, y, s)) ||
        self_mask2(V, G) != (self_mask(v, t) & self_mask(w, s)))
        return fail("mask2", V, X, G, 0);
    /* every form that solves both tests is matched */
    if ((pair_mask(v, x, t) & pair_mask(w, y, s)) && !last_any(V, last_keys(X, G)))
        return fail("pair", V, X, G, 0);
    if ((self_mask(v, t) & self_mask(w, s)) && !last_any_self(V, G)) return fail("self", V, G, 0, 0);
    /* one test in both halves: a match is a form that solves it */
    if (last_any(v * 0x10001u, last_keys(x * 0x10001u, t * 0x10001u)) != (pair_mask(v, x, t) != 0))
        return fail("one test", v, x, t, 0);
    return 0;
}

static bool copy_or_zero(uint32_t u)
{
    const uint32_t op = UOP_OP(u), a = UOP_A(u), b = UOP_B(u);
    if (op == PCA_OP_LDI) return UOP_IMM(u) == 0;
    if (op == PCA_OP_ADDI) return false;
    if (a == b) return op == PCA_OP_AND || op == PCA_OP_OR || op == PCA_OP_XOR || op == PCA_OP_SUB;
    if (b == 0) return op != PCA_OP_SHL && op != PCA_OP_SHR && op != PCA_OP_ASR;
    if (a == 0) return op != PCA_OP_SUB && op != PCA_OP_MUL;
    return false;
}

int main()
{
    std::vector<uint32_t> edge;
    for (int k = 0; k < 16; k++)
        for (int d = -2; d <= 2; d++) {
            edge.push_back(((1u << k) + d) & 0xFFFF);
            edge.push_back((0u - (1u << k) + d) & 0xFFFF);
        }
    std::mt19937 g(7);
    auto word = [&] { return (uint32_t)(g() & 0xFFFF) >> (g() % 3 ? 0 : g() % 16); };
    for (uint32_t x : edge)
        for (uint32_t t : edge)
            for (int i = 0; i < 200; i++)
                if (keys(i < 160 ? edge[i] : word(), x, t, word(), edge[g() % 160], edge[g() % 160]))
                    return 1;
    /* every v for words x, t: the keys are exact, not a sample */
    for (int i = 0; i < 300; i++) {
        const uint32_t x = i & 1 ? word() : edge[g() % edge.size()];
        const uint32_t t = i & 2 ? pair_value(g() % 13, word(), x) : edge[g() % edge.size()];
        const LastKeys k = last_keys(x * 0x10001u, t * 0x10001u);
        for (uint32_t v = 0; v < 65536; v++)
            if (last_any(v * 0x10001u, k) != (pair_mask(v, x, t) != 0))
                return fail("one test", v, x, t, 1);
    }
    for (int i = 0; i < 2000000; i++)
    {
        /* both tests solved by one form of (v, x), or the targets left alone */
        const uint32_t v = word(), x = word(), w = word(), y = word(), f = g() % 13;
        const bool one = i & 1;
        if (keys(v, x, one ? pair_value(f, v, x) : word(), w, y, one ? pair_value(f, w, y) : word()))
            return 1;
        if (keys(v, x, self_value(f % 12, v), w, y, self_value(f % 12, w))) return 1;
    }

    const GenTables &gt = gen_tables();
    for (uint32_t m = 0; m < 128; m++) {
        std::map<uint32_t, int> form;
        std::vector<uint32_t> regs;
        for (uint32_t r = 1; r < 8; r++)
            if (m >> (r - 1) & 1) regs.push_back(r);
        for (size_t i = 0; i < regs.size(); i++)
            for (size_t j = i; j < regs.size(); j++)
                for (uint32_t f = 0; f < (i == j ? (uint32_t)kSelfForms : (uint32_t)kPairForms); f++)
                    form[form_uop(i == j ? kKindSelf : kKindPair, f, regs[i], regs[j])]++;
        for (uint32_t f = 0; f < kLdiForms; f++) form[form_uop(kKindLdi, f, 0, 0)]++;
        std::set<uint32_t> classes(gt.vc_uop.begin() + gt.vc_off[m],
                                   gt.vc_uop.begin() + gt.vc_off[m + 1]);
        for (uint32_t u : classes)
            if (!form.count(u) && !copy_or_zero(u)) return fail("class without a form", m, u, 0, 0);
        for (auto &p : form) {
            if (p.second != 1) return fail("class of two forms", m, p.first, 0, 0);
            if (!classes.count(p.first)) return fail("form without a class", m, p.first, 0, 0);
            if (UOP_OP(p.first) != PCA_OP_LDI && copy_or_zero(p.first))
                return fail("a form that copies", m, p.first, 0, 0);
        }
        /* the LDI classes' places, and each class's candidates by destination */
        const uint32_t nvc = gt.vc_off[m + 1] - gt.vc_off[m];
        for (uint32_t f = 0; f < kLdiForms; f++)
            if (gt.vc_uop[gt.vc_off[m] + nvc - 6 * regs.size() - kLdiForms + f] !=
                form_uop(kKindLdi, f, 0, 0))
                return fail("LDI class", m, f, 0, 0);
        uint32_t listed = 0;
        for (uint32_t c = 0; c < nvc; c++)
            for (uint32_t rd = 0; rd < 8; rd++) {
                const uint32_t i = gt.cand_of[(gt.vc_off[m] + c) * 8 + rd];
                if (i == 0xFFFF) continue;
                listed++;
                if (gt.cand_vc[gt.cand_off[m] + i] != c ||
                    UOP_RD(gt.cand_uop[gt.cand_off[m] + i]) != rd)
                    return fail("candidate of a class", m, c, rd, i);
            }
        if (listed != gt.cand_off[m + 1] - gt.cand_off[m]) return fail("candidates", m, listed, 0, 0);
        /* the last instruction of (v, x) and of v alone, by its pair entry */
        for (uint32_t v : regs) {
            std::set<uint32_t> seen;
            for (uint32_t x : regs)
                for (uint32_t f = 0; f < (x == v ? (uint32_t)kSelfForms : (uint32_t)kPairForms); f++) {
                    uint32_t ab, k, found = 0;
                    if (x == v) self_entry(f, v, ab, k);
                    else pair_entry(f, v, x, ab, k);
                    const uint32_t i = m * 8 + v;
                    const uint32_t e = k == 9 ? gt.pr_off[i + 1] - 6 + f - kFAddi
                                              : gt.pr_off[i] + gt.pr_at[i * 64 + ab];
                    if (e < gt.pr_off[i + 1] && (gt.pr[e] & 63u) == ab && gt.pr[e] >> (6 + k) & 1u) {
                        found++;
                        const uint32_t c = gt.pr_cls[e * 10 + k], u = gt.vc_uop[gt.vc_off[m] + c];
                        if (u != form_uop(x == v ? kKindSelf : kKindPair, f, v, x) || !seen.insert(c).second)
                            return fail("entry of another class", m, v, x, f);
                    }
                    if (found != 1) return fail("entries of a form", m, v, x, f);
                }
        }
    }
    puts("ok");
    return 0;
}
"""


def test_value_forms_on_the_host(tmp_path):
    build_engine()
    src, exe = tmp_path / "forms.cpp", tmp_path / "forms"
    src.write_text(PROGRAM)
    lib = os.path.join(LIBDIR, "libpcagb.so")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, str(src), lib,
                        f"-Wl,-rpath,{LIBDIR}", "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
