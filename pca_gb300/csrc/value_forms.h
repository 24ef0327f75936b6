/*
 * value_forms.h -- the values a position can write, and the middle values that
 * solve a target (shared by the suffix kernels and the host tests).
 *
 * What an instruction writes does not depend on its destination, so a
 * position is a set of values over the registers in reach: for two registers
 * x, y the thirteen of kPairForms (nine ALU ops, the four that do not
 * commute in both orders), for one register the twelve of kSelfForms (the ops
 * of it with itself, its negative, six ADDI), and the LDI immediates. The
 * generator's other classes write a copy of a register (ADD/OR/XOR with r0,
 * AND/OR of a register with itself) or zero (AND or a shift with r0,
 * XOR/SUB of a register with itself). Neither can be a middle or a last
 * instruction of a solving program at a depth K >= 3: with it left out and
 * its register (for zero: r0) read instead, K-1 instructions reach the
 * target, and K-1 was searched without a solution. (A target of zeros was
 * found at depth 1. An ADDI reads no r0, but what it makes of zero is found by
 * depth 2: -1, -2 and -3; the positive ones are LDI immediates. So a depth-2
 * search from the root has to try zero as its middle.) So they are not
 * enumerated.
 *
 * A solving program's every write is read (the read rule of scan_last), so
 * the value v of the instruction before the last is an operand of the last
 * one. With the other operand x and the target t of a test fixed, the v that
 * solve it are known in closed form (LastKeys): t - x, t + x, x - t and t ^ x
 * for ADD, SUB in both orders and XOR; v & x == t; v | x == t; a residue for
 * MUL (the inverse of x's odd part); the low or high bits of v for the shifts
 * of v; a set of v & 15 for the shifts of x by v. Deciding a middle value
 * against all thirteen last instructions with x is eleven compares, where
 * evaluating them takes about forty instructions; with two tests to a word
 * the same compares decide both.
 */
#ifndef PCA_VALUE_FORMS_H
#define PCA_VALUE_FORMS_H

#include "pca_isa.h"

#if defined(__CUDACC__)
#define PCA_UNROLL _Pragma("unroll")
#else
#define PCA_UNROLL
#endif

namespace pcagb {

/* highest set bit (-1 for zero), trailing zeros of a nonzero word, the
   sixteen bits of x reversed, x >> (s mod 32) */
PCA_HD int top_bit(uint32_t x)
{
#if defined(__CUDA_ARCH__)
    return 31 - __clz((int)x);
#else
    return x ? 31 - __builtin_clz(x) : -1;
#endif
}

PCA_HD uint32_t low_bit(uint32_t x)
{
#if defined(__CUDA_ARCH__)
    return (uint32_t)__ffs((int)x) - 1u;
#else
    return (uint32_t)__builtin_ctz(x);
#endif
}

PCA_HD uint32_t rev16(uint32_t x)
{
#if defined(__CUDA_ARCH__)
    return __brev(x) >> 16;
#else
    uint32_t r = 0;
    for (int i = 0; i < 16; i++) r |= (x >> i & 1u) << (15 - i);
    return r;
#endif
}

PCA_HD uint32_t shr_wrap(uint32_t x, uint32_t s)
{
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(x, 0u, s);
#else
    return x >> (s & 31u);
#endif
}

/* values of two registers */
enum PairForm : uint32_t {
    kFAdd, kFSub, kFRsub, kFMul, kFAnd, kFOr, kFXor, kFShl, kFRshl, kFShr, kFRshr, kFAsr, kFRasr,
    kPairForms
};
/* values of one register; the ADDI immediates follow kFAddi */
enum SelfForm : uint32_t { kFDbl, kFSqr, kFShlS, kFShrS, kFAsrS, kFNeg, kFAddi, kSelfForms = 12 };
constexpr uint32_t kLdiForms = 12;
/* groups of middle values: of two registers, of one, of none */
enum FormKind : uint32_t { kKindPair, kKindSelf, kKindLdi };

PCA_HD uint32_t addi_imm(uint32_t k)   /* k = 0..5: -1, 1, -2, 2, -3, 3 */
{
    const uint32_t m = (k >> 1) + 1;
    return k & 1 ? m : (0u - m);
}

PCA_HD uint32_t ldi_imm(uint32_t k)    /* 0..5, 8, 16, 32, 64, 128, 255 */
{
    return k < 6 ? k : k == 11 ? 255u : 8u << (k - 6);
}

PCA_HD uint32_t asr16(uint32_t x, uint32_t s)
{
    return (uint32_t)((int32_t)(int16_t)(uint16_t)x >> s) & 0xFFFFu;
}

PCA_HD uint32_t pair_value(uint32_t f, uint32_t x, uint32_t y)
{
    switch (f) {
    case kFAdd: return (x + y) & 0xFFFFu;
    case kFSub: return (x - y) & 0xFFFFu;
    case kFRsub: return (y - x) & 0xFFFFu;
    case kFMul: return (x * y) & 0xFFFFu;
    case kFAnd: return x & y;
    case kFOr: return x | y;
    case kFXor: return x ^ y;
    case kFShl: return (x << (y & 15u)) & 0xFFFFu;
    case kFRshl: return (y << (x & 15u)) & 0xFFFFu;
    case kFShr: return x >> (y & 15u);
    case kFRshr: return y >> (x & 15u);
    case kFAsr: return asr16(x, y & 15u);
    default: return asr16(y, x & 15u);
    }
}

PCA_HD uint32_t self_value(uint32_t f, uint32_t x)
{
    switch (f) {
    case kFDbl: return (x + x) & 0xFFFFu;
    case kFSqr: return (x * x) & 0xFFFFu;
    case kFShlS: return (x << (x & 15u)) & 0xFFFFu;
    case kFShrS: return x >> (x & 15u);
    case kFAsrS: return asr16(x, x & 15u);
    case kFNeg: return (0u - x) & 0xFFFFu;
    default: return (x + addi_imm(f - kFAddi)) & 0xFFFFu;
    }
}

PCA_HD uint32_t form_value(uint32_t kind, uint32_t f, uint32_t x, uint32_t y)
{
    return kind == kKindPair ? pair_value(f, x, y) : kind == kKindSelf ? self_value(f, x) : ldi_imm(f);
}

/* which forms of (v, x) give t: bit f */
PCA_HD uint32_t pair_mask(uint32_t v, uint32_t x, uint32_t t)
{
    uint32_t h = 0;
    PCA_UNROLL
    for (uint32_t f = 0; f < kPairForms; f++) h |= (uint32_t)(pair_value(f, v, x) == t) << f;
    return h;
}

PCA_HD uint32_t self_mask(uint32_t v, uint32_t t)
{
    uint32_t h = 0;
    PCA_UNROLL
    for (uint32_t f = 0; f < kSelfForms; f++) h |= (uint32_t)(self_value(f, v) == t) << f;
    return h;
}

/* the shifts s for which x >> s == t (bit s of sixteen) */
PCA_HD uint32_t shift_set(uint32_t x, uint32_t t)
{
    const int lx = top_bit(x), lt = top_bit(t);   /* -1 for zero */
    if (t == 0) return (0xFFFFu << (lx + 1)) & 0xFFFFu;
    const int d = lx - lt;
    return d >= 0 && (x >> d) == t ? 1u << d : 0u;
}

/* ---- two tests to a word ----------------------------------------------------
   The low and the high half of a word hold a register's values on two
   tests. One compare of words is then one form on both tests. */
PCA_HD uint32_t add2(uint32_t x, uint32_t y)
{
#if defined(__CUDA_ARCH__)
    uint32_t r;
    asm("add.u16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
    return r;
#else
    return ((x + y) & 0xFFFFu) | ((x & 0xFFFF0000u) + (y & 0xFFFF0000u));
#endif
}

PCA_HD uint32_t sub2(uint32_t x, uint32_t y) { return ~add2(~x, y); }

/* the low half of lo and the high half of hi */
PCA_HD uint32_t halves(uint32_t lo, uint32_t hi)
{
#if defined(__CUDA_ARCH__)
    return __byte_perm(lo, hi, 0x7610);
#else
    return (lo & 0xFFFFu) | (hi & 0xFFFF0000u);
#endif
}

/* the high halves of lo and hi */
PCA_HD uint32_t high_halves(uint32_t lo, uint32_t hi)
{
#if defined(__CUDA_ARCH__)
    return __byte_perm(lo, hi, 0x7632);
#else
    return (lo >> 16) | (hi & 0xFFFF0000u);
#endif
}

PCA_HD uint32_t mul2(uint32_t x, uint32_t y)
{
    return halves(x * y, ((x >> 16) * (y >> 16)) << 16);
}

PCA_HD uint32_t shl2(uint32_t x, uint32_t y)
{
    return halves(x << (y & 15u), (x & 0xFFFF0000u) << (y >> 16 & 15u));
}

PCA_HD uint32_t shr2(uint32_t x, uint32_t y)
{
    return halves((x & 0xFFFFu) >> (y & 15u), x >> (y >> 16 & 15u));
}

PCA_HD uint32_t asr2(uint32_t x, uint32_t y)
{
    return high_halves((uint32_t)((int32_t)(x << 16) >> (y & 15u)),
                       (uint32_t)((int32_t)x >> (y >> 16 & 15u)));
}

PCA_HD uint32_t pair_value2(uint32_t f, uint32_t x, uint32_t y)
{
    switch (f) {
    case kFAdd: return add2(x, y);
    case kFSub: return sub2(x, y);
    case kFRsub: return sub2(y, x);
    case kFMul: return mul2(x, y);
    case kFAnd: return x & y;
    case kFOr: return x | y;
    case kFXor: return x ^ y;
    case kFShl: return shl2(x, y);
    case kFRshl: return shl2(y, x);
    case kFShr: return shr2(x, y);
    case kFRshr: return shr2(y, x);
    case kFAsr: return asr2(x, y);
    default: return asr2(y, x);
    }
}

PCA_HD uint32_t self_value2(uint32_t f, uint32_t x)
{
    switch (f) {
    case kFDbl: return add2(x, x);
    case kFSqr: return mul2(x, x);
    case kFShlS: return shl2(x, x);
    case kFShrS: return shr2(x, x);
    case kFAsrS: return asr2(x, x);
    case kFNeg: return sub2(0, x);
    default: return add2(x, (addi_imm(f - kFAddi) & 0xFFFFu) * 0x10001u);
    }
}

/* which forms give t on both tests */
PCA_HD uint32_t pair_mask2(uint32_t v, uint32_t x, uint32_t t)
{
    uint32_t h = 0;
    PCA_UNROLL
    for (uint32_t f = 0; f < kPairForms; f++) h |= (uint32_t)(pair_value2(f, v, x) == t) << f;
    return h;
}

PCA_HD uint32_t self_mask2(uint32_t v, uint32_t t)
{
    uint32_t h = 0;
    PCA_UNROLL
    for (uint32_t f = 0; f < kSelfForms; f++) h |= (uint32_t)(self_value2(f, v) == t) << f;
    return h;
}

/* The v for which some form of (v, x) gives t, on two tests at once: v equals
   add, sub, rsub or xr; v & x == t; v | x == t; (v & mulm) == mulc;
   (v & shlm) == shlc (v << x); (v & shrm) == shrc (v >> x of either kind, so
   the two tests may differ in the kind); bit v & 15 of vset0 and vset1 (x
   shifted by v, any of the three kinds on each test; sixteen bits, twice). A
   condition that no v meets on a test compares with a bit outside its
   mask. Every v that solves both tests by one form matches. */
struct LastKeys {
    uint32_t x, t, add, sub, rsub, xr, mulm, mulc, shlm, shlc, shrm, shrc, vset0, vset1;
};

/* one test's mulm | mulc << 16, shlm | shlc << 16, shrm | shrc << 16, vset */
PCA_HD void last_keys1(uint32_t x, uint32_t t, uint32_t &mul, uint32_t &shl, uint32_t &shr,
                       uint32_t &vset)
{
    /* v x = t mod 2^16: with x = 2^z o, o odd, t must be a multiple of 2^z
       and v = (t / 2^z) / o mod 2^(16 - z); o's inverse by Newton's step
       y (2 - o y), which doubles the correct low bits (5 of (3 o) ^ 2) */
    const uint32_t z = x ? low_bit(x) : 16u;
    const uint32_t o = x >> z;
    uint32_t y = (3u * o) ^ 2u;
    y *= 2u - o * y;
    y *= 2u - o * y;
    const uint32_t mm = 0xFFFFu >> z;
    mul = mm | ((t & ((1u << z) - 1u)) ? 0x8000u : ((t >> z) * y) & mm) << 16;
    const uint32_t s = x & 15u;
    shl = (0xFFFFu >> s) | ((t & ((1u << s) - 1u)) ? 0x8000u : t >> s) << 16;
    const uint32_t c = (t << s) & 0xFFFFu;
    shr = ((0xFFFFu << s) & 0xFFFFu) | ((c >> s) == t || asr16(c, s) == t ? c : 1u) << 16;
    /* x << v is x >> v of the reversed words; the arithmetic shift of a
       negative x is the logical one of the complements */
    const bool neg = x >> 15;
    vset = shift_set(x, t) | shift_set(rev16(x), rev16(t)) |
           shift_set(neg ? x ^ 0xFFFFu : x, neg ? t ^ 0xFFFFu : t);
    vset |= vset << 16;
}

PCA_HD LastKeys last_keys(uint32_t x, uint32_t t)
{
    LastKeys k;
    k.x = x;
    k.t = t;
    k.add = sub2(t, x);
    k.sub = add2(t, x);
    k.rsub = sub2(x, t);
    k.xr = t ^ x;
    uint32_t m0, l0, r0, m1, l1, r1;
    last_keys1(x & 0xFFFFu, t & 0xFFFFu, m0, l0, r0, k.vset0);
    last_keys1(x >> 16, t >> 16, m1, l1, r1, k.vset1);
    k.mulm = halves(m0, m1 << 16);
    k.mulc = high_halves(m0, m1);
    k.shlm = halves(l0, l1 << 16);
    k.shlc = high_halves(l0, l1);
    k.shrm = halves(r0, r1 << 16);
    k.shrc = high_halves(r0, r1);
    return k;
}

PCA_HD bool last_any(uint32_t v, const LastKeys &k)
{
    return (v == k.add) | (v == k.sub) | (v == k.rsub) | (v == k.xr) | ((v & k.x) == k.t) |
           ((v | k.x) == k.t) | ((v & k.mulm) == k.mulc) | ((v & k.shlm) == k.shlc) |
           ((v & k.shrm) == k.shrc) |
           (shr_wrap(k.vset0, v) & shr_wrap(k.vset1, v >> 16) & 1u);
}

/* the same for the last instructions of v alone (the ADDI as one range, v
   itself among it, the same immediate on both tests) */
PCA_HD bool last_any_self(uint32_t v, uint32_t t)
{
    const uint32_t d = sub2(t, v);
    return (add2(v, v) == t) | (add2(v, t) == 0u) | (mul2(v, v) == t) | (shl2(v, v) == t) |
           (shr2(v, v) == t) | (asr2(v, v) == t) |
           ((d >> 16) == (d & 0xFFFFu) && ((d + 3u) & 0xFFFFu) <= 6u);
}

/* ---- the classes of a form ------------------------------------------------- */

/* the op of an operand-pair entry's opmask bit */
PCA_HD uint32_t pair_op(uint32_t k)
{
    switch (k) {
    case 0: return PCA_OP_ADD;
    case 1: return PCA_OP_SUB;
    case 2: return PCA_OP_MUL;
    case 3: return PCA_OP_AND;
    case 4: return PCA_OP_OR;
    case 5: return PCA_OP_XOR;
    case 6: return PCA_OP_SHL;
    case 7: return PCA_OP_SHR;
    case 8: return PCA_OP_ASR;
    default: return PCA_OP_ADDI;
    }
}

/* operand-pair entry of the last instruction `f` of (register v, register x):
   a | b << 3 and the op's bit */
PCA_HD void pair_entry(uint32_t f, uint32_t v, uint32_t x, uint32_t &ab,
                                           uint32_t &k)
{
    const uint32_t lo = v < x ? v : x, hi = v < x ? x : v;
    switch (f) {
    case kFAdd: k = 0; break;
    case kFSub: case kFRsub: k = 1; break;
    case kFMul: k = 2; break;
    case kFAnd: k = 3; break;
    case kFOr: k = 4; break;
    case kFXor: k = 5; break;
    case kFShl: case kFRshl: k = 6; break;
    case kFShr: case kFRshr: k = 7; break;
    default: k = 8; break;
    }
    const bool forward = f == kFSub || f == kFShl || f == kFShr || f == kFAsr;
    const bool backward = f == kFRsub || f == kFRshl || f == kFRshr || f == kFRasr;
    ab = forward ? (v | x << 3) : backward ? (x | v << 3) : (lo | hi << 3);
}

/* the same for the forms of one register */
PCA_HD void self_entry(uint32_t f, uint32_t v, uint32_t &ab, uint32_t &k)
{
    ab = v | v << 3;
    switch (f) {
    case kFDbl: k = 0; break;
    case kFSqr: k = 2; break;
    case kFShlS: k = 6; break;
    case kFShrS: k = 7; break;
    case kFAsrS: k = 8; break;
    case kFNeg: k = 1; ab = v << 3; break;
    default: k = 9; ab = v; break;   /* ADDI: the entry holds the register in a */
    }
}

/* micro-op of a middle form without its destination (an ADDI keeps it) */
PCA_HD uint32_t form_uop(uint32_t kind, uint32_t f, uint32_t x, uint32_t y)
{
    if (kind == kKindLdi) return PCA_OP_LDI | ldi_imm(f) << 16;
    uint32_t ab, k;
    if (kind == kKindPair) pair_entry(f, x, y, ab, k);
    else self_entry(f, x, ab, k);
    if (k == 9) return PCA_OP_ADDI | x << 5 | x << 8 | (addi_imm(f - kFAddi) & 0xFFu) << 16;
    return pair_op(k) | (ab & 7u) << 8 | (ab >> 3) << 11;
}

}  // namespace pcagb

#endif
