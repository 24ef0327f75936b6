/*
 * suffix_forms.cuh -- the suffix kernels over value forms (included by
 * engine_kernels.cuh): the last position, a lane per prefix, and the last two, a
 * lane per state.
 */
#pragma once

namespace pcagb {

/* ---- shared parts of the lane kernels -------------------------------------- */

/* Index of the entry of the operand-pair list of (mask m, register r) that
   holds op bit k on operands ab (value_forms.h); ADDI entries (k = 9) are the
   list's last six, in immediate order. */
__device__ __forceinline__ uint32_t pair_index(uint32_t m, uint32_t r, uint32_t ab, uint32_t k,
                                               uint32_t addi)
{
    const uint32_t i = m * 8 + r;
    return k == 9 ? c_pr_off_g[i + 1] - 6 + addi : c_pr_off_g[i] + c_pr_at[i * 64 + ab];
}

/* Value class (in mask m's list) of a middle form on registers x, y. */
__device__ __forceinline__ uint32_t form_class(uint32_t m, uint32_t kind, uint32_t f, uint32_t x,
                                               uint32_t y)
{
    if (kind == kKindLdi)   /* the classes end with the LDI's, then six ADDI a register */
        return c_vc_off[m + 1] - c_vc_off[m] - 6 * (uint32_t)__popc(m) - kLdiForms + f;
    uint32_t ab, k;
    if (kind == kKindPair) pair_entry(f, x, y, ab, k);
    else self_entry(f, x, ab, k);
    return c_pr_cls[(uint64_t)pair_index(m, x, ab, k, f - kFAddi) * 10 + k];
}

/* Records the last instructions `forms` (of register v with x, or of v
   alone) that solve after a write to register v left mask m. Each lane
   records its own. */
__device__ __forceinline__ void record_last(const SolBuf &S, uint32_t m, uint32_t v, uint32_t x,
                                            bool self, uint32_t forms, uint64_t q, uint32_t m1,
                                            uint32_t m2)
{
    while (forms) {
        const uint32_t f = (uint32_t)__ffs((int)forms) - 1u;
        forms &= forms - 1;
        uint32_t ab, k;
        if (self) self_entry(f, v, ab, k);
        else pair_entry(f, v, x, ab, k);
        const uint32_t c = c_pr_cls[(uint64_t)pair_index(m, v, ab, k, f - kFAddi) * 10 + k];
        record_solution(S, q, m1, m2, c, m);
    }
}

/* ---- suffix depth 1 --------------------------------------------------------- */

/* The last position, a lane per prefix. The last instruction reads the
 * prefix's last write v; the other operand is one of the prefix's other
 * live registers or v itself. A lane holds its prefix's 64-byte probe
 * (r0..r7 on the first four tests) in registers and evaluates the thirteen
 * forms of (v, x) for each live x, and the twelve of v, two tests to a word:
 * on the first test (FT = 1), on the first two (2), or on all four (3).
 * What is left is checked on every test by the warp (lane = test), from the
 * level's columns or, on a lean level, from the parent's columns and the
 * prefix's last instruction.
 *
 * Bound: integer issue (59% active), about 700 warp instructions for 32
 * prefixes, and 75 bytes of HBM a prefix. 5.3M prefixes of is_power2: 0.52 ms
 * walking the generator's operand pairs from memory (2,000 instructions, the
 * operands looked up in shared memory), 0.21-0.28 ms by forms, 0.15 ms where
 * the targets are less alike (popcount); reading the prefixes takes 0.06. */
template <int TPC, int FT>
__global__ void __launch_bounds__(kThreads, 4)
k_suffix_lanes(LevelDev P, TaskDev task, SolBuf S, PrefixRange R, LeanDev lean)
{
    const int lane = threadIdx.x & 31;
    const uint64_t nt = (uint64_t)gridDim.x * kThreads;
    const uint64_t n_round = (R.count + 31) & ~31ull;
    uint32_t nev = 0;   /* this lane's prefixes' readable classes (the evaluation count) */
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < n_round; i += nt) {
        uint64_t q = ~0ull;
        if (i < R.count) {
            q = R.order ? (uint64_t)R.order[R.begin + i] : R.begin + i;
            if (q >= P.n) q = ~0ull;   /* orders are checked on the host; never index outside */
        }
        uint32_t tid = 0, live = 0, w0 = 0, T = 0, t01 = 0, t23 = 0;
        uint4 pr[4] = {};
        if (q != ~0ull) {
            tid = P.task[q];
            live = P.live[q];
            w0 = P.rdl[q];
            const uint4 *pp = reinterpret_cast<const uint4 *>(P.probe + q * 32);
#pragma unroll
            for (int h = 0; h < 4; h++) pr[h] = pp[h];
            if (task.active[tid] && w0) {
                T = (uint32_t)task.T[tid];
                nev += __ldg(c_ev_sd1 + ((live >> 1) & 127u) * 8 + w0);
                const uint4 tt = *reinterpret_cast<const uint4 *>(task.target + tid * 32);
                t01 = FT >= 2 && T >= 2 ? tt.x | tt.y << 16 : tt.x * 0x10001u;
                t23 = tt.z | (T >= 4 ? tt.w : tt.z) << 16;
            } else {
                w0 = 0;
            }
        }
        /* register r's words (two tests each); a lone test fills both halves */
        auto word = [&](uint32_t r, int p) -> uint32_t {
            const uint4 w = r < 2 ? pr[0] : r < 4 ? pr[1] : r < 6 ? pr[2] : pr[3];
            const uint32_t u = p ? (r & 1 ? w.w : w.y) : (r & 1 ? w.z : w.x);
            const bool lone = p ? T < 4 : FT == 1 || T < 2;
            return lone ? __byte_perm(u, 0, 0x1010) : u;
        };
        const uint32_t v01 = word(w0, 0), v23 = FT >= 3 ? word(w0, 1) : 0u;
        /* x = 1..7: another live register; 8: v alone */
#pragma unroll 1
        for (uint32_t x = 1; x <= 8; x++) {
            const bool self = x == 8;
            const bool on = w0 && (self || (((live >> x) & 1u) && x != w0));
            if (!__any_sync(0xFFFFFFFFu, on)) continue;
            uint32_t hits = 0;
            if (on) {
                hits = self ? self_mask2(v01, t01) : pair_mask2(v01, word(x, 0), t01);
                if (FT >= 3 && T >= 3 && hits)
                    hits &= self ? self_mask2(v23, t23) : pair_mask2(v23, word(x, 1), t23);
            }
            uint32_t bal = __ballot_sync(0xFFFFFFFFu, hits != 0);
            while (bal) {
                const int L = __ffs(bal) - 1;
                bal &= bal - 1;
                const unsigned long long qL = __shfl_sync(0xFFFFFFFFu, (unsigned long long)q, L);
                const uint32_t tidL = __shfl_sync(0xFFFFFFFFu, tid, L);
                const uint32_t liveL = __shfl_sync(0xFFFFFFFFu, live, L);
                const uint32_t wL = __shfl_sync(0xFFFFFFFFu, w0, L);
                const uint32_t hL = __shfl_sync(0xFFFFFFFFu, hits, L);
                const int TL = task.T[tidL];
                uint32_t ok = ~0u;
                if (lane < TL) {
                    uint32_t a, b;
                    const uint32_t xr = self ? wL : (uint32_t)x;
                    if (!lean.up_regs) {
                        a = P.regs[(qL * 8 + wL) * TPC + lane];
                        b = P.regs[(qL * 8 + xr) * TPC + lane];
                    } else {
                        /* a lean level: the prefix's registers are its
                           parent's but for the one its last instruction wrote */
                        const uint64_t pL = P.parent[qL];
                        const uint32_t uL = c_cand_uop[c_cand_off[(lean.up_live[pL] >> 1) & 127u] +
                                                       lean.cidx[qL]];
                        const uint16_t *up = lean.up_regs + pL * 8 * TPC + lane;
                        a = pca_alu(UOP_OP(uL), up[UOP_A(uL) * TPC], up[UOP_B(uL) * TPC],
                                    UOP_IMM(uL)) & 0xFFFFu;
                        b = up[xr * TPC];
                    }
                    const uint32_t tg = task.target[tidL * 32 + lane];
                    ok = self ? self_mask(a, tg) : pair_mask(a, b, tg);
                }
                const uint32_t forms = __reduce_and_sync(0xFFFFFFFFu, ok) & hL;
                if (forms >> lane & 1u)   /* a form a lane */
                    record_last(S, (liveL >> 1) & 127u, wL, (uint32_t)x, self, 1u << lane, qL, 0, 0);
            }
        }
    }
    /* the stage's evaluation count (k_count_evals' sum for these prefixes) */
    flush_evals(S, nev, lane);
}

/* One warp's shared memory in k_suffix_states, a column per lane: the
   registers by position ([tests 0-1, 2-3][position], two tests to a word),
   the keys of the current x on either pair of tests, and the middle values
   of the current group. The values pass through shared memory so that the
   compare loop is one short body: thirteen unrolled copies of it ran at a
   quarter of the issue rate, waiting for instruction fetches. */
constexpr int kStatesWarps = 4;
struct StatesWarp {
    uint32_t V[2][7][32];
    uint32_t key[2][14][32];
    uint32_t val[kPairForms][32];
};

__device__ __forceinline__ void store_keys(uint32_t (&K)[14][32], const LastKeys &k, int lane)
{
    K[0][lane] = k.x; K[1][lane] = k.t; K[2][lane] = k.add; K[3][lane] = k.sub;
    K[4][lane] = k.rsub; K[5][lane] = k.xr; K[6][lane] = k.mulm; K[7][lane] = k.mulc;
    K[8][lane] = k.shlm; K[9][lane] = k.shlc; K[10][lane] = k.shrm; K[11][lane] = k.shrc;
    K[12][lane] = k.vset0; K[13][lane] = k.vset1;
}

__device__ __forceinline__ LastKeys load_keys(const uint32_t (&K)[14][32], int lane)
{
    return LastKeys{K[0][lane], K[1][lane], K[2][lane], K[3][lane], K[4][lane],
                    K[5][lane], K[6][lane], K[7][lane], K[8][lane], K[9][lane],
                    K[10][lane], K[11][lane], K[12][lane], K[13][lane]};
}

/* ---- suffix depths 2 and 3 -------------------------------------------------- */

/* The last two positions, a lane per state: at suffix depth 2 the state is a
 * prefix, at depth 3 a prefix and one of its first middles (per_prefix of
 * them to a prefix, the lane computing the middle's value on the probe's
 * four tests). A lane keeps its state's registers on those tests in shared
 * memory by position: first A and B, the registers that the remaining two
 * instructions must read (the last write; at depth 3 the prefix's last write
 * too when the first middle does not read it), then the other live ones.
 *
 * For every operand x of the last instruction (each live register, and the
 * middle's value itself) the lane forms the keys of the first two tests'
 * targets once and compares every middle value with them (LastKeys: two
 * tests to a word). A middle that
 * reads all of A and B meets every x; one that leaves one of them unread
 * only that register; one that leaves both none. A value that matches is
 * evaluated in its lane, form by form, on up to five more tests (a target
 * of few values lets whole families pass the probe's: 0.5% of is_power2's
 * values pass four), then on every test by the warp (lane = test), and one
 * that no test rules out is expanded to the candidates that write it (destinations and rules as k_suffix).
 *
 * Work items are 32 states and one of 2^slices_log2 shares of their
 * (x, group) pairs, so small levels fill the GPU too.
 *
 * Bound: integer issue, the ALU pipe first (72% of it at 59% issue). 5.3M
 * prefixes, suffix depth 2, every middle and last instruction: 376 ms with a
 * lane per middle that evaluates the operand pairs, 3.4 ms here (popcount;
 * is_power2, whose values pass more tests, 425 and 5.3); depth 3 from 100K
 * two-input states' parents 3.3 -> 0.2 ms. */
template <int TPC, int SD>
__global__ void __launch_bounds__(kStatesWarps * 32, 8)
k_suffix_states(LevelDev P, TaskDev task, SolBuf S, uint32_t per_prefix, uint32_t slices_log2,
                PrefixRange R)
{
    static_assert(SD == 2 || SD == 3, "suffix depths 2 and 3");
    __shared__ StatesWarp sw[kStatesWarps];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    StatesWarp &W = sw[wib];
    const uint64_t nw = (uint64_t)gridDim.x * kStatesWarps;
    const uint64_t total = R.count * per_prefix;
    const uint64_t items = ((total + 31) >> 5) << slices_log2;
    const uint32_t slices = 1u << slices_log2;
    const uint32_t *ev_mid = c_ev_mid + (task.dedup_mid ? 128 * 64 : 0);
    unsigned long long nev = 0;
    for (uint64_t it = (uint64_t)blockIdx.x * kStatesWarps + wib; it < items; it += nw) {
        const uint32_t slice = (uint32_t)it & (slices - 1);
        const uint64_t i = (it >> slices_log2) * 32 + lane;
        uint64_t q = ~0ull;
        uint32_t i1 = 0;
        if (i < total) {
            const uint64_t qi = SD == 3 ? i / per_prefix : i;
            if (SD == 3) i1 = (uint32_t)(i - qi * per_prefix);
            q = R.order ? (uint64_t)R.order[R.begin + qi] : R.begin + qi;
            if (q >= P.n) q = ~0ull;   /* orders are checked on the host; never index outside */
        }
        uint32_t tid = 0, mask = 0, A = 0, B = 0, T = 0, u1 = 0;
        bool valid = false;
        if (q != ~0ull) {
            tid = P.task[q];
            mask = (P.live[q] >> 1) & 127u;
            A = P.rdl[q];
            valid = task.active[tid] != 0;
            if (SD == 3 && valid) {
                const uint32_t cb = c_cand_off[mask];
                valid = i1 < c_cand_off[mask + 1] - cb;
                if (valid) {
                    u1 = c_cand_uop[cb + i1];
                    const uint32_t rd = UOP_RD(u1);
                    B = A && !uop_reads(u1, A) ? A : 0u;
                    if ((task.dedup_mid && (u1 >> 31)) || (B && rd == B)) valid = false;
                    mask |= 1u << (rd - 1);
                    A = rd;
                }
            }
        }
        uint32_t t01 = 0, t23 = 0, L = 0, regs_at = 0;   /* regs_at: register of each position, 4 bits */
        __syncwarp();
        if (valid) {
            T = (uint32_t)task.T[tid];
            const uint4 tt = *reinterpret_cast<const uint4 *>(task.target + tid * 32);
            t01 = tt.x | (T >= 2 ? tt.y : tt.x) << 16;
            t23 = tt.z | (T >= 4 ? tt.w : tt.z) << 16;
            if (slice == 0) nev += __ldg(ev_mid + (mask * 8 + A) * 8 + B);
            const uint2 *pp = reinterpret_cast<const uint2 *>(P.probe + q * 32);
            uint2 w1 = make_uint2(0, 0);
            if (SD == 3) {
                const uint2 a = pp[UOP_A(u1)], b = pp[UOP_B(u1)];
                const uint32_t op = UOP_OP(u1), imm = UOP_IMM(u1);
                w1.x = pca_alu(op, a.x & 0xFFFFu, b.x & 0xFFFFu, imm) |
                       pca_alu(op, a.x >> 16, b.x >> 16, imm) << 16;
                w1.y = pca_alu(op, a.y & 0xFFFFu, b.y & 0xFFFFu, imm) |
                       pca_alu(op, a.y >> 16, b.y >> 16, imm) << 16;
            }
            uint32_t next = (A ? 1u : 0u) + (B ? 1u : 0u);
#pragma unroll
            for (uint32_t r = 1; r < 8; r++) {
                if (!((mask >> (r - 1)) & 1u)) continue;
                const uint2 w = SD == 3 && r == A ? w1 : pp[r];
                const uint32_t p = r == A ? 0u : r == B ? 1u : next++;
                regs_at |= r << (4 * p);
                /* a lone test fills both halves */
                W.V[0][p][lane] = T >= 2 ? w.x : halves(w.x, w.x << 16);
                W.V[1][p][lane] = T >= 4 ? w.y : halves(w.y, w.y << 16);
            }
            L = (uint32_t)__popc(mask);
        }
        __syncwarp();
        if (!__any_sync(0xFFFFFFFFu, valid)) continue;
        const uint32_t Lm = __reduce_max_sync(0xFFFFFFFFu, L);
        const bool hasA = A != 0, hasB = B != 0;
        uint32_t job = 0;
        /* x: the last instruction's other operand; Lm = the middle's value */
        for (uint32_t x = 0; x <= Lm; x++) {
            const bool self = x == Lm;
            uint32_t have = 0;   /* pairs of tests whose keys for this x are formed */
            /* groups of middle values: registers a <= b; a == Lm: the LDI */
            for (uint32_t a = 0; a <= Lm; a++)
                for (uint32_t b = a; b < max(Lm, a + 1); b++) {
                    if ((job++ & (slices - 1)) != slice) continue;
                    const uint32_t kind = a == Lm ? kKindLdi : a == b ? kKindSelf : kKindPair;
                    const bool ua = hasA && a != 0;                  /* A, B unread */
                    const bool ub = hasB && a != 1 && b != 1;
                    bool ok = valid && (kind == kKindLdi || b < L) && (self || x < L);
                    if (ua || ub) ok = ok && !self && !(ua && ub) && x == (ua ? 0u : 1u);
                    /* forms some last instruction takes to the target, on
                       tests 0-1, then on 2-3 where any is left */
                    const uint32_t all = kind == kKindPair   ? (1u << kPairForms) - 1u
                                         : kind == kKindSelf ? (1u << kSelfForms) - 1u
                                                             : (1u << kLdiForms) - 2u;   /* 0 is r0 */
                    uint32_t hits = ok ? all : 0u;
#pragma unroll 1
                    for (uint32_t p = 0; p < 2; p++) {
                        if (!__any_sync(0xFFFFFFFFu, hits)) break;
                        const uint32_t tp = p ? t23 : t01;
                        if (!self && have <= p) {
                            have = p + 1;
                            store_keys(W.key[p], last_keys(W.V[p][x][lane], tp), lane);
                        }
                        if (kind == kKindPair) {
                            const uint32_t wa = W.V[p][a][lane], wb = W.V[p][b][lane];
#pragma unroll
                            for (uint32_t f = 0; f < kPairForms; f++)
                                W.val[f][lane] = pair_value2(f, wa, wb);
                        } else if (kind == kKindSelf) {
                            const uint32_t wa = W.V[p][a][lane];
#pragma unroll
                            for (uint32_t f = 0; f < kSelfForms; f++)
                                W.val[f][lane] = self_value2(f, wa);
                        } else {
#pragma unroll
                            for (uint32_t f = 0; f < kLdiForms; f++)
                                W.val[f][lane] = ldi_imm(f) * 0x10001u;
                        }
                        uint32_t h = 0;
                        if (self) {
#pragma unroll 1
                            for (uint32_t f = 0; f < kPairForms; f++)
                                h |= (uint32_t)last_any_self(W.val[f][lane], tp) << f;
                        } else {
                            const LastKeys key = load_keys(W.key[p], lane);
#pragma unroll 1
                            for (uint32_t f = 0; f < 12; f += 3)
                                h |= ((uint32_t)last_any(W.val[f][lane], key) |
                                      (uint32_t)last_any(W.val[f + 1][lane], key) << 1 |
                                      (uint32_t)last_any(W.val[f + 2][lane], key) << 2)
                                     << f;
                            if (kind == kKindPair)
                                h |= (uint32_t)last_any(W.val[12][lane], key) << 12;
                        }
                        if (p == 0 || T >= 3) hits &= h;
                    }
                    uint32_t fm = __reduce_or_sync(0xFFFFFFFFu, hits);
                    /* rare: a few tests in the lane, last form by last form:
                       the first, then those past the probe */
                    while (fm) {
                        const uint32_t f = (uint32_t)__ffs((int)fm) - 1u;
                        fm &= fm - 1;
                        uint32_t lf = 0;   /* last forms this lane's value passes */
                        if ((hits >> f) & 1u) {
                            lf = ~0u;
                            const uint16_t *col = P.regs + q * 8 * TPC;
                            const uint32_t ra = regs_at >> (4 * a) & 7u, rb = regs_at >> (4 * b) & 7u;
                            const uint32_t rx = self ? 0u : regs_at >> (4 * x) & 7u;
#pragma unroll 1
                            for (uint32_t k = 0; k < min(T, 8u) && lf; k = k ? k + 1 : 4) {
                                uint32_t va = col[ra * TPC + k], vb = col[rb * TPC + k];
                                uint32_t vx = col[rx * TPC + k];
                                if (SD == 3) {
                                    const uint32_t c1 =
                                        pca_alu(UOP_OP(u1), col[UOP_A(u1) * TPC + k],
                                                col[UOP_B(u1) * TPC + k], UOP_IMM(u1));
                                    if (ra == A) va = c1;
                                    if (rb == A) vb = c1;
                                    if (rx == A) vx = c1;
                                }
                                const uint32_t mv = form_value(kind, f, va, vb);
                                const uint32_t tk = task.target[tid * 32 + k];
                                lf &= self ? self_mask(mv, tk) : pair_mask(mv, vx, tk);
                            }
                        }
                        uint32_t bal = __ballot_sync(0xFFFFFFFFu, lf != 0);
                        while (bal) {
                            /* every test by the warp, lane = test */
                            const int j = __ffs((int)bal) - 1;
                            bal &= bal - 1;
                            const unsigned long long qj =
                                __shfl_sync(0xFFFFFFFFu, (unsigned long long)q, j);
                            const uint32_t tj = __shfl_sync(0xFFFFFFFFu, tid, j);
                            const uint32_t Tj = __shfl_sync(0xFFFFFFFFu, T, j);
                            const uint32_t Aj = __shfl_sync(0xFFFFFFFFu, A, j);
                            const uint32_t uj = __shfl_sync(0xFFFFFFFFu, u1, j);
                            const uint32_t at = __shfl_sync(0xFFFFFFFFu, regs_at, j);
                            const uint32_t ra = at >> (4 * a) & 7u, rb = at >> (4 * b) & 7u;
                            const uint32_t rx = self ? 0u : at >> (4 * x) & 7u;
                            uint32_t pass = ~0u;
                            if ((uint32_t)lane < Tj) {
                                const uint16_t *col = P.regs + qj * 8 * TPC + lane;
                                uint32_t va = col[ra * TPC], vb = col[rb * TPC], vx = col[rx * TPC];
                                if (SD == 3) {
                                    const uint32_t c1 = pca_alu(UOP_OP(uj), col[UOP_A(uj) * TPC],
                                                                col[UOP_B(uj) * TPC], UOP_IMM(uj));
                                    if (ra == Aj) va = c1;
                                    if (rb == Aj) vb = c1;
                                    if (rx == Aj) vx = c1;
                                }
                                const uint32_t mv = form_value(kind, f, va, vb);
                                const uint32_t tg = task.target[tj * 32 + lane];
                                pass = self ? self_mask(mv, tg) : pair_mask(mv, vx, tg);
                            }
                            const uint32_t forms = __reduce_and_sync(0xFFFFFFFFu, pass) &
                                                   __shfl_sync(0xFFFFFFFFu, lf, j);
                            const uint32_t mj = __shfl_sync(0xFFFFFFFFu, mask, j);
                            const uint32_t Bj = __shfl_sync(0xFFFFFFFFu, B, j);
                            const uint32_t ij = __shfl_sync(0xFFFFFFFFu, i1, j);
                            if (!forms) continue;
                            /* a solving (value, last instruction): the
                               candidates that write it, lane = destination */
                            const uint32_t c = c_vc_off[mj] + form_class(mj, kind, f, ra, rb);
                            const uint32_t ch = lane >= 1 && lane < 8 ? c_cand_of[c * 8 + lane]
                                                                      : 0xFFFFu;
                            if (ch == 0xFFFFu) continue;
                            const uint32_t u = c_cand_uop[c_cand_off[mj] + ch];
                            const uint32_t rd = (uint32_t)lane;
                            const uint32_t need2 = Aj && !uop_reads(u, Aj)   ? Aj
                                                   : Bj && !uop_reads(u, Bj) ? Bj : 0u;
                            if ((task.dedup_mid && (u >> 31)) || (need2 && rd == need2) ||
                                (!self && rx == rd))
                                continue;
                            record_last(S, (mj | (1u << (rd - 1))) & 127u, rd, rx, self, forms, qj,
                                        SD == 3 ? ij : ch, SD == 3 ? ch : 0u);
                        }
                    }
                }
        }
    }
    flush_evals(S, nev, lane);
}

}  // namespace pcagb
