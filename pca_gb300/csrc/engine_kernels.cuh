/*
 * engine_kernels.cuh -- CUDA kernels of the PCA-16 exhaustive engine.
 *
 * Search levels. Level d holds the distinct states reached by d kernel
 * instructions (level 0 = the task root). A state is stored column-major:
 * regs[n][8][TP] (u16, r0's column kept as zeros), flags[n][TP], live[n],
 * plus the back pointer (parent rank, candidate index) that rebuilds its
 * program. TP is 16 or 32 (test count rounded up), and test slots >= T are
 * zero in every state.
 *
 * Level expansion (the OEP kernel): one warp per parent. It forms each value
 * class of the parent's candidates once, a lane a class: the new column (two
 * tests to a word), its hash, its flags as bit planes and the column's exact
 * id; then a lane takes a child (class, destination), whose 64-bit hash comes
 * from the parent's per-column hashes, and inserts a 64-bit slot
 *   [tag: hash bits 40..63][ref + 1: 40 bits]
 * into an open-addressed HBM table, ref = parent_rank << 12 | candidate.
 * On a tag match the two child states are compared exactly, by the ids of
 * their columns or, on levels too small or too large for ids, column by
 * column (every register of every test, flags, and live when it is part of
 * the key), so a hash collision can never merge two different states. Among
 * equal states the smallest ref wins (atomicCAS loop), which is the first
 * child in the reference's DFS order -- the representative the reference's
 * DFS pruner keeps (tools/enumerate.c:379-384). Children that can never be
 * that representative are not inserted at all: same-state siblings of an
 * earlier candidate (bit 31 of the device micro-op), children overwriting a
 * dead-able unread write (deadable_writes) and LDI swaps (ldi_swap); each
 * has an equal state with a smaller ref, so the winners do not change.
 *
 * The insert keeps a bitmap of the winners beside the table, indexed by the
 * child's linear index (child_off[parent] + candidate); its bits are ranked
 * by a scan and the winners written out in that order, so every level stays
 * in DFS order.
 *
 * Suffix kernels. The last instruction's value does not depend on its
 * destination (except ADDI), so only value classes are evaluated, and only
 * those that read the last write (the read rule in scan_last). Large levels
 * take a lane per prefix or per state, by value forms (suffix_forms.cuh);
 * here are the warp-per-prefix kernels of roots, small levels and forced
 * shapes: one lane per operand pair, every op of the pair evaluated on the
 * first two tests at once, each survivor checked on all tests by the warp
 * (lane t taking test t, __all_sync deciding), the middle instructions of
 * suffix depths 2 and 3 in spare shared-memory columns 8 and 9.
 */
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "pca_isa.h"
#include "scan.cuh"
#include "value_forms.h"

namespace pcagb {

constexpr int kWarpsPerBlock = 8;
constexpr int kThreads = kWarpsPerBlock * 32;
constexpr uint64_t kRefMask = (1ull << 40) - 1;
constexpr uint32_t kMaxProbes = 1u << 16;

/* status flags set by kernels (bounded loops that ran out) */
constexpr uint32_t kStatusTableFull = 1u;
constexpr uint32_t kStatusRefOverflow = 2u;

/* Candidate tables, uploaded once per device. */
__constant__ uint32_t c_cand_off[129];
__constant__ uint32_t c_vc_off[129];
__constant__ const uint32_t *c_cand_uop;   /* bit 31: a same-state duplicate of an earlier candidate */
__constant__ const uint32_t *c_vc_uop;
__constant__ const uint16_t *c_vc_first;   /* first candidate index per class */
__constant__ const uint8_t *c_vc_n;        /* candidates per class */
__constant__ uint32_t c_vchunk_off[129];   /* op-uniform runs of value classes */
__constant__ const uint32_t *c_vchunks;    /* first class << 8 | classes (at most 32) */
__constant__ const uint2 *c_cand_k;        /* micro-op and value class of each candidate */
__constant__ const uint32_t *c_cand_off_g; /* c_cand_off in global memory (lanes of different masks) */
__constant__ const uint16_t *c_kid;        /* [class][8] candidate of the class by destination;
                                              0xFFFF: none, or a same-state duplicate */
__constant__ uint32_t c_vcr_off[128 * 8 + 1]; /* [mask*8 + r]: classes reading r */
__constant__ const uint32_t *c_vcr_uop;    /* their micro-ops */
__constant__ uint32_t c_pr_off[128 * 8 + 1];  /* [mask*8 + r]: the same, by operand pair */
__constant__ const uint32_t *c_pr;         /* a | b << 3 | opmask << 6 | imm << 16 */
__constant__ const uint16_t *c_pr_cls;     /* [entry][10] class index per opmask bit */
__constant__ uint32_t c_pr_ev[128 * 8];    /* [mask*8 + r]: class evaluations of its pair list */
__constant__ const uint32_t *c_ev_sd1;     /* the same in global memory, [mask*8 + 0] = all classes */
__constant__ const uint16_t *c_pr_at;      /* GenTables::pr_at, cand_of */
__constant__ const uint16_t *c_cand_of;
__constant__ const uint32_t *c_ev_mid;     /* [dedup_mid][mask][A][B]: evaluations of the last two
                                              positions from a state of that mask whose registers
                                              A and B (0: none) they must read */
__constant__ const uint32_t *c_pr_off_g;   /* c_pr_off in global memory (lanes of different masks) */

/* Per-task parameters of a batch: device arrays indexed by task id. A
   state's task id travels with it through the levels; states of different
   tasks never compare equal. */
struct TaskDev {
    const int32_t *T;          /* tests of each task */
    const uint32_t *target;    /* [task][32] expected outputs */
    const uint8_t *active;     /* task still searched at the current depth */
    int key_live;              /* OEP key includes live */
    int dedup_mid;             /* OEP on: a suffix's middle instruction that
                                  repeats an earlier sibling's state is skipped */
};

struct LevelDev {
    const uint16_t *regs;   /* [n][8][TP] */
    const uint8_t *flags;   /* [n][TP] */
    const uint8_t *live;    /* [n] */
    const uint16_t *task;   /* [n] */
    const uint64_t *child_off; /* [n+1] */
    uint64_t n;
    const uint8_t *rdl;     /* [n] register the state's last instruction wrote (0: root) */
    const uint32_t *parent; /* [n] rank of the parent in the level above */
    const uint8_t *own;     /* [n] registers whose last write is unread and dead-able (below);
                               bit 0: the last instruction is an LDI */
    const uint8_t *twin;    /* [n] 1: an earlier state of the level has the same registers,
                               live mask and task (k_twins) */
    const uint16_t *probe;  /* [n][8][4] r0..r7 on the first four tests, 64 bytes a state */
};

/* A lean level (k_materialize_probe: links and probes, no register block)
   reaches its states' registers through their parents: the level above's
   registers and liveness, and the lean level's own candidate indices.
   up_regs == nullptr: the level is a full one. */
struct LeanDev {
    const uint16_t *up_regs;   /* [n_up][8][TP] */
    const uint8_t *up_live;    /* [n_up] */
    const uint16_t *cidx;      /* [n] candidate index of each state in its parent's list */
};

struct LevelOut {
    uint16_t *regs;
    uint8_t *flags;
    uint8_t *live;
    uint16_t *task;
    uint32_t *parent;
    uint16_t *cidx;
    uint8_t *rdl;
    uint8_t *own;
    uint16_t *probe;
};

/* ---- hashing (a multiply-rotate chain; the table compares full states, so
        the hash only has to spread well) -------------------------------- */

__device__ __forceinline__ uint64_t fmix64(uint64_t x)
{
    x ^= x >> 33;
    x *= 0xFF51AFD7ED558CCDull;
    x ^= x >> 33;
    x *= 0xC4CEB9FE1A85EC53ull;
    x ^= x >> 33;
    return x;
}

__device__ __forceinline__ uint64_t chain(uint64_t h, uint64_t w)
{
    h = (h ^ w) * 0x9E3779B97F4A7C15ull;
    return (h << 27) | (h >> 37);
}

__device__ __forceinline__ uint64_t col_final(uint32_t r, uint64_t h)
{
    return fmix64(h + (uint64_t)r * 0xD6E8FEB86659FD93ull);
}

__device__ __forceinline__ uint64_t live_final(uint32_t live)
{
    return fmix64(0x5851F42D4C957F2Dull ^ live);
}

__device__ __forceinline__ uint64_t task_final(uint32_t task)
{
    return fmix64(0x9E3779B97F4A7C15ull * (task + 1));
}

/* a column's hash, two tests to a word */
template <int TPC>
__device__ __forceinline__ uint64_t hash_column(const uint32_t *col)
{
    uint64_t h = 0x243F6A8885A308D3ull;
#pragma unroll
    for (int t = 0; t < TPC / 2; t += 2) h = chain(h, (uint64_t)col[t + 1] << 32 | col[t]);
    return h;
}

/* Reads: does micro-op u read register r (1..7)? */
__device__ __forceinline__ bool uop_reads(uint32_t u, uint32_t r)
{
    return UOP_A(u) == r || UOP_B(u) == r;
}

/* Dead writes. In a state's path, a write to register w that no later
   instruction has read yet, made by an instruction z that is not the first
   kept sibling writing w (the lowest-ranked kept child of z's parent that
   writes w), is dead-able: a child y that is not an LDI and overwrites w
   without reading it reaches a state (registers, y's flags, live) that the
   same path with the first sibling in z's place reaches too, by a smaller
   ref (every instruction after z is the same candidate under the same
   liveness mask, and none reads w). Such a child is never the DFS-first
   representative, so the insert kernel skips it and the table's winners,
   and every level, are unchanged. A state keeps these registers in `own`
   (writes older than its last instruction); its last write is dead-able
   when the state is not the first kept sibling writing it (fcr_up, the
   first-child ranks of the level above). */
__device__ __forceinline__ uint32_t deadable_writes(const LevelDev &P, const uint32_t *fcr_up,
                                                    uint64_t q)
{
    if (!fcr_up) return 0;
    uint32_t W = P.own[q] & 0xFEu;
    const uint32_t w = P.rdl[q];
    if (w && fcr_up[(uint64_t)P.parent[q] * 8 + w] != (uint32_t)q) W |= 1u << w;
    return W;
}

/* LDI swaps. When a state's last instruction is an LDI (bit 0 of `own`)
   writing register y, a child x that neither reads nor writes y reaches the
   state of the path with x and the LDI in the other order (the LDI keeps
   the flags, so both end with x's). That path is the smaller ref when x
   comes first in the generator's order: every ALU op precedes every LDI,
   and an LDI precedes another when its register is lower. Such a child is
   never the DFS-first representative; the insert kernel skips it. */
__device__ __forceinline__ bool ldi_swap(uint32_t u, uint32_t last_ldi_reg)
{
    if (!last_ldi_reg) return false;
    const uint32_t op = UOP_OP(u), rd = UOP_RD(u);
    if (rd == last_ldi_reg || uop_reads(u, last_ldi_reg)) return false;
    if (op == PCA_OP_LDI) return rd < last_ldi_reg;
    return op != PCA_OP_ADDI;
}

/* ---- shared-memory view of one state per warp ---------------------------- */

template <int TPC>
struct WarpState {
    uint32_t R[10][TPC + 1];  /* columns r0..r7 + 2 spare; +1 word pad */
    uint32_t F[TPC];
    uint64_t colh[8];         /* colh[r] = col_final(r, hash(col r)), r >= 1 */
};

/* ---- set-up of a batch -------------------------------------------------- */

/* One task's root as the host hands it over, tests in the caller's order. */
struct __align__(16) RootIn {
    uint16_t regs[32][8];
    uint16_t target[32];
    uint8_t flags[32];
    uint8_t live;
    uint8_t T;
};

/* Where the set-up writes the batch's per-task arrays. */
struct SetupOut {
    int32_t *T;
    uint32_t *target;   /* [task][32], in the engine's test order */
    uint16_t *io;       /* [task][3][32] inputs 0 and 1, target, in that order */
    uint8_t *order;     /* [task][32] the caller's test at each place */
    uint32_t *status;
    unsigned long long *evals;
};

/* Level 0 and the test order of every task: a block per task.
 *
 * The suffix kernels reject almost every value on a state's first tests, so
 * these are chosen to reject: each next test is the one that the fewest
 * (state, last instruction) pairs pass among the pairs that pass every test
 * chosen before; once no pair is left the choice starts over, until the
 * probe's four tests are chosen (a deeper state's values pass the first ones
 * more often than the sample's, so each should reject well by itself). Ties
 * go to a target not met yet: a constant passes equal targets together. The
 * other tests keep the caller's order. A permutation of the tests changes no
 * result of the search.
 *
 * The states are drawn (the same ones for every call) two instructions from
 * the root, 17 a round, a warp each; the pairs are their classes that read
 * the second write. One round serves a search of depth 4, whose last stage
 * is over in a quarter of a millisecond; a deeper one takes eight, for on a
 * target of few values one round's sample is too small: of is_power2's
 * values at depth 5, one in 700 passed four tests chosen on 17 states and one
 * in 50,000 tests chosen on 136 (a fifth of the stage's time).
 *
 * Bound: latency, a warp's walk over some fifty classes a round. On the host
 * such a choice took 50-300 us a task, most of the time of a small solve and
 * nine tenths of a batch of 256. */
constexpr int kSetupWarps = 17;
constexpr uint32_t kSetupPairs = 224;   /* passing pairs kept a warp */

template <int TPC>
__global__ void __launch_bounds__(kSetupWarps * 32)
k_setup(const RootIn *in, uint32_t rounds, LevelOut L0, uint8_t *twin, SetupOut out)
{
    __shared__ RootIn root;
    __shared__ uint16_t st[kSetupWarps][8][32];
    __shared__ uint32_t sp[kSetupWarps][kSetupPairs];
    __shared__ uint32_t cnt[32], alive;
    __shared__ uint8_t order[32];
    const uint32_t i = blockIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    static_assert(sizeof(RootIn) % 16 == 0, "copied in 16-byte pieces");
    for (uint32_t k = threadIdx.x; k < sizeof(RootIn) / 16; k += blockDim.x)
        reinterpret_cast<uint4 *>(&root)[k] = reinterpret_cast<const uint4 *>(in + i)[k];
    if (threadIdx.x < 32) cnt[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t T = root.T, live = root.live;
    const uint32_t target = (uint32_t)lane < T ? root.target[lane] : 0x10000u;
    uint16_t (&R)[8][32] = st[w];
    uint32_t *pairs = sp[w], np = 0;
    for (uint32_t rd = 0; rd < rounds; rd++) {
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 8; r++) R[r][lane] = root.regs[lane][r];
        uint32_t m = (live >> 1) & 127u, last = 0;
#pragma unroll
        for (uint32_t k = 0; k < 2; k++) {
            const uint32_t nc = c_cand_off[m + 1] - c_cand_off[m];
            const uint32_t pick = ((rd * kSetupWarps + w) * 2 + k + 1) * 2654435761u;
            const uint32_t u = c_cand_uop[c_cand_off[m] + __umulhi(pick, nc)];
            const uint16_t v = (uint16_t)pca_alu(UOP_OP(u), R[UOP_A(u)][lane], R[UOP_B(u)][lane],
                                                 UOP_IMM(u));
            last = UOP_RD(u);
            m |= 1u << (last - 1);
            R[last][lane] = v;   /* each lane reads only its own test */
        }
        const uint32_t v0 = c_vcr_off[m * 8 + last], nv = c_vcr_off[m * 8 + last + 1] - v0;
        for (uint32_t b = 0; b < nv; b += 32) {
            const uint32_t mine = b + lane < nv ? c_vcr_uop[v0 + b + lane] : 0u;
            const uint32_t n = min(32u, nv - b);
            for (uint32_t k = 0; k < n; k++) {
                const uint32_t u = __shfl_sync(0xFFFFFFFFu, mine, k);
                const uint32_t v = pca_alu(UOP_OP(u), R[UOP_A(u)][lane], R[UOP_B(u)][lane],
                                           UOP_IMM(u));
                const uint32_t pass = __ballot_sync(0xFFFFFFFFu, v == target);
                if (pass && np < kSetupPairs) {
                    if (lane == 0) pairs[np] = pass;
                    np++;
                }
            }
        }
    }
    __syncwarp();
    uint32_t used = 0, need = 0;   /* chosen tests; those since the last start */
    for (uint32_t r = 0; r < 4 && r < T; r++) {
        uint32_t c = 0, any = 0;
        for (uint32_t k = 0; k < np; k++) {
            const uint32_t p = pairs[k];
            if ((p & need) != need) continue;
            any = 1;
            c += p >> lane & 1u;
        }
        if (threadIdx.x == 0) alive = 0;
        __syncthreads();
        if (c) atomicAdd(&cnt[lane], c);
        if (any && lane == 0) alive = 1;
        __syncthreads();
        if (!alive && need) {
            /* every pair ruled out: start over (cnt is all zero) */
            need = 0;
            r--;
            __syncthreads();
            continue;
        }
        if (w == 0) {
            bool fresh = true;
            for (uint32_t k = 0; k < r; k++) fresh &= root.target[order[k]] != target;
            uint32_t key = (uint32_t)lane < T && !(used >> lane & 1u)
                               ? (cnt[lane] * 2 + (fresh ? 0u : 1u)) * 32 + lane : ~0u;
            key = __reduce_min_sync(0xFFFFFFFFu, key);
            if (lane == 0) order[r] = (uint8_t)(key & 31u);
        }
        __syncthreads();
        if (threadIdx.x < 32) cnt[threadIdx.x] = 0;
        used |= 1u << order[r];
        need |= 1u << order[r];
        __syncthreads();
    }
    if (w == 0) {
        const uint32_t rest = ~used & (T >= 32 ? ~0u : (1u << T) - 1u);
        if (rest >> lane & 1u)
            order[__popc(used) + __popc(rest & ((1u << lane) - 1u))] = (uint8_t)lane;
    }
    __syncthreads();
    /* level 0, in the engine's test order */
    for (uint32_t k = threadIdx.x; k < 8 * TPC; k += blockDim.x) {
        const uint32_t r = k / TPC, t = k % TPC;
        const uint16_t v = r && t < T ? root.regs[order[t]][r] : (uint16_t)0;
        L0.regs[(uint64_t)i * 8 * TPC + k] = v;
        if (t < 4) L0.probe[(uint64_t)i * 32 + r * 4 + t] = v;
    }
    if (w == 0) {
        const uint32_t o = (uint32_t)lane < T ? order[lane] : 0u;
        const bool in_t = (uint32_t)lane < T;
        if (lane < TPC) L0.flags[(uint64_t)i * TPC + lane] = in_t ? root.flags[o] : (uint8_t)0;
        out.target[i * 32 + lane] = in_t ? root.target[o] : 0u;
        uint16_t *io = out.io + (uint64_t)i * 96 + lane;
        io[0] = in_t ? root.regs[o][1] : (uint16_t)0;
        io[32] = in_t ? root.regs[o][2] : (uint16_t)0;
        io[64] = in_t ? root.target[o] : (uint16_t)0;
        out.order[i * 32 + lane] = (uint8_t)o;
        if (lane == 0) {
            L0.live[i] = (uint8_t)live;
            L0.task[i] = (uint16_t)i;
            L0.parent[i] = 0;
            L0.cidx[i] = 0;
            L0.rdl[i] = 0;
            L0.own[i] = 0;
            twin[i] = 0;
            out.T[i] = (int32_t)T;
            if (i == 0) {
                *out.status = 0;
                *out.evals = 0;
            }
        }
    }
}

/* ---- level expansion: insert every child into the exact table ------------ */

/* ---- flags of a state as four planes -----------------------------------------
   A plane (Z, N, C, V) holds one flag on every test, a bit a test: test t at
   bit TPC/2 - 1 - t/2, the odd tests sixteen higher (two tests of a word
   enter a plane by one shift and add). */
template <int TPC>
__device__ __forceinline__ uint32_t plane_bit(int t)
{
    return (uint32_t)(TPC / 2 - 1 - (t >> 1) + 16 * (t & 1));
}

/* the bits of the tests below T */
template <int TPC>
__device__ __forceinline__ uint32_t plane_mask(int T)
{
    const uint32_t even = (uint32_t)(T + 1) / 2, odd = (uint32_t)T / 2;
    return ((1u << even) - 1u) << (TPC / 2 - even) | ((1u << odd) - 1u) << (TPC / 2 - odd) << 16;
}

/* One warp's shared memory in the insert kernel: its parent (two tests to a
   word, a row stride of TPC / 2 + 1 words so that lanes reading different
   operand columns of one test hit different banks), the column, flags and
   hashes of each value class of the current chunk (a class a lane), and the
   chunk's children. */
template <int TPC>
struct InsertState {
    uint4 flagsA[33];                      /* [class] Z, N, C, V planes; [32]: the parent's */
    uint64_t colA[32][TPC / 4 + 1];        /* [class][four tests] */
    uint64_t colh[8];                      /* colh[r] = col_final(r, hash(col r)), r >= 1 */
    uint64_t hA[32], hfA[32];              /* [class] the column's and the flags' hash */
    uint32_t idA[32], ids[8];              /* column ids: the classes', the parent's registers' */
    uint32_t R[8][TPC / 2 + 1];
    uint8_t F[TPC];
    uint8_t kids[256];                     /* class << 3 | destination */
};

/* A class's new column and flags, two tests to a word; the op is a template
   parameter: a warp takes a run of classes that share one, so the switch is
   resolved at compile time and the lanes never diverge on it. Leaves the
   column and the planes in shared memory and returns their hashes (tests >= T
   are zero in both). */
template <int TPC, int OP>
__device__ __forceinline__ void class_values(InsertState<TPC> &ws, uint32_t ra, uint32_t rb,
                                             uint32_t imm, int T, int lane, uint64_t &h,
                                             uint64_t &hf)
{
    const uint32_t imm2 = OP == PCA_OP_LDI ? imm * 0x10001u
                                           : (uint32_t)(uint16_t)(int16_t)(int8_t)(uint8_t)imm * 0x10001u;
    constexpr bool kCarry = OP == PCA_OP_ADD || OP == PCA_OP_SUB || OP == PCA_OP_MUL ||
                            OP == PCA_OP_ADDI;
    constexpr bool kOver = kCarry && OP != PCA_OP_MUL;
    uint32_t Z = 0, N = 0, C = 0, V = 0;
    h = 0x243F6A8885A308D3ull;
#pragma unroll 1
    for (int i = 0; i < TPC / 4; i++) {
        uint32_t v[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t a = ws.R[ra][2 * i + k];
            const uint32_t b = OP == PCA_OP_ADDI ? imm2 : ws.R[rb][2 * i + k];
            uint32_t r, c = 0, o = 0;
            if constexpr (OP == PCA_OP_ADD || OP == PCA_OP_ADDI) {
                r = add2(a, b);
                c = (a & b) | ((a | b) & ~r);
                o = ~(a ^ b) & (a ^ r);
            } else if constexpr (OP == PCA_OP_SUB) {
                r = sub2(a, b);
                c = ~((~a & b) | ((~a | b) & r));   /* no borrow */
                o = (a ^ b) & (a ^ r);
            } else if constexpr (OP == PCA_OP_MUL) {
                const uint32_t p0 = (a & 0xFFFFu) * (b & 0xFFFFu), p1 = (a >> 16) * (b >> 16);
                r = halves(p0, p1 << 16);
                c = (p0 > 0xFFFFu ? 0x8000u : 0u) | (p1 > 0xFFFFu ? 0x80000000u : 0u);
            } else if constexpr (OP == PCA_OP_AND) r = a & b;
            else if constexpr (OP == PCA_OP_OR) r = a | b;
            else if constexpr (OP == PCA_OP_XOR) r = a ^ b;
            else if constexpr (OP == PCA_OP_SHL) r = shl2(a, b);
            else if constexpr (OP == PCA_OP_SHR) r = shr2(a, b);
            else if constexpr (OP == PCA_OP_ASR) r = asr2(a, b);
            else r = imm2;
            if constexpr (OP != PCA_OP_LDI) {
                const uint32_t nz = ((r & 0x7FFF7FFFu) + 0x7FFF7FFFu) | r;
                Z = Z * 2 + (~nz >> 15 & 0x10001u);
                N = N * 2 + (r >> 15 & 0x10001u);
                if constexpr (kCarry) C = C * 2 + (c >> 15 & 0x10001u);
                if constexpr (kOver) V = V * 2 + (o >> 15 & 0x10001u);
            }
            v[k] = r;
        }
        const int left = T - 4 * i;   /* tests of this word */
        if (left < 4) {
            v[0] = left >= 2 ? v[0] : left == 1 ? v[0] & 0xFFFFu : 0u;
            v[1] = left == 3 ? v[1] & 0xFFFFu : 0u;
        }
        const uint64_t w = (uint64_t)v[1] << 32 | v[0];
        ws.colA[lane][i] = w;
        h = chain(h, w);
    }
    uint4 f;
    if constexpr (OP == PCA_OP_LDI) {
        f = ws.flagsA[32];
    } else {
        const uint32_t m = plane_mask<TPC>(T);
        f = make_uint4(Z & m, N & m, C & m, V & m);
    }
    ws.flagsA[lane] = f;
    hf = chain(chain(0x13198A2E03707344ull, (uint64_t)f.y << 32 | f.x), (uint64_t)f.w << 32 | f.z);
}

template <int TPC>
__device__ __forceinline__ void class_values_any(uint32_t op, InsertState<TPC> &ws, uint32_t ra,
                                                 uint32_t rb, uint32_t imm, int T, int lane,
                                                 uint64_t &h, uint64_t &hf)
{
    switch (op) {
    case PCA_OP_ADD: class_values<TPC, PCA_OP_ADD>(ws, ra, rb, imm, T, lane, h, hf); break;
    case PCA_OP_SUB: class_values<TPC, PCA_OP_SUB>(ws, ra, rb, imm, T, lane, h, hf); break;
    case PCA_OP_MUL: class_values<TPC, PCA_OP_MUL>(ws, ra, rb, imm, T, lane, h, hf); break;
    case PCA_OP_AND: class_values<TPC, PCA_OP_AND>(ws, ra, rb, imm, T, lane, h, hf); break;
    case PCA_OP_OR: class_values<TPC, PCA_OP_OR>(ws, ra, rb, imm, T, lane, h, hf); break;
    case PCA_OP_XOR: class_values<TPC, PCA_OP_XOR>(ws, ra, rb, imm, T, lane, h, hf); break;
    case PCA_OP_SHL: class_values<TPC, PCA_OP_SHL>(ws, ra, rb, imm, T, lane, h, hf); break;
    case PCA_OP_SHR: class_values<TPC, PCA_OP_SHR>(ws, ra, rb, imm, T, lane, h, hf); break;
    case PCA_OP_ASR: class_values<TPC, PCA_OP_ASR>(ws, ra, rb, imm, T, lane, h, hf); break;
    case PCA_OP_LDI: class_values<TPC, PCA_OP_LDI>(ws, ra, rb, imm, T, lane, h, hf); break;
    default: class_values<TPC, PCA_OP_ADDI>(ws, ra, rb, imm, T, lane, h, hf); break;
    }
}

/* ---- exact column ids --------------------------------------------------------
   Every distinct register column met while a level is expanded (its states'
   registers, its classes' values) gets an id from an exact table: a column is
   written to `cols` under a fresh id, then published in a slot [tag 24][id + 1:
   40]; a tag match is settled by comparing the whole column. Equal ids are
   equal columns and equal columns have equal ids, so two children are the
   same state when their register ids and flag planes are: a lane compares its
   own, where comparing the columns takes the warp and a hundred instructions
   a pair. The table and the arrays live only while the level is expanded. */
struct IdDev {
    unsigned long long *tab;   /* [mask + 1] slots; null: no ids (compare columns) */
    uint64_t mask;
    uint64_t *cols;            /* [cap][TPC / 4] */
    uint32_t cap;
    uint32_t *next;            /* ids given out, kIdBatch at a time to a warp */
    uint32_t *ids;             /* [n][8] of the level's registers; r0's place: task << 8 | live */
    uint32_t *cls_id;          /* [n][stride] of its classes' columns */
    uint4 *cls_flags;          /* [n][stride] planes of its classes */
    uint32_t stride;
};
constexpr uint32_t kIdBatch = 64;
constexpr uint32_t kStatusColumns = 4u;    /* out of ids or slots: expand without them */

__device__ __forceinline__ unsigned long long load_acquire(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

/* A warp's ids not yet used: [at, end). */
struct IdPool {
    uint32_t at = 0, end = 0;
};

/* The id of this lane's column (col, hash h) where `want`; all lanes call it. */
template <int TPC>
__device__ __forceinline__ uint32_t intern(const IdDev &D, const uint64_t *col, uint64_t h,
                                           bool want, IdPool &pool, uint32_t *status, int lane)
{
    const uint64_t H = fmix64(h);
    const unsigned long long tag = H >> 40;
    uint64_t idx = H & D.mask;
    uint32_t mine = ~0u, id = 0, probes = 0;
    bool done = !want;
    while (__any_sync(0xFFFFFFFFu, !done)) {
        unsigned long long s = done ? 1ull : load_acquire(&D.tab[idx]);
        const bool need = !done && s == 0 && mine == ~0u;
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, need);
        if (bal) {
            const uint32_t n = __popc(bal);
            if (pool.end - pool.at < n) {   /* the rest of the old batch is dropped */
                uint32_t b = 0;
                if (lane == 0) b = atomicAdd(D.next, kIdBatch);
                pool.at = __shfl_sync(0xFFFFFFFFu, b, 0);
                pool.end = pool.at + kIdBatch;
            }
            if (need) {
                mine = pool.at + __popc(bal & ((1u << lane) - 1u));
                if (mine >= D.cap) {
                    atomicOr(status, kStatusColumns);
                    done = true;
                } else {
                    uint4 *dst = reinterpret_cast<uint4 *>(D.cols + (uint64_t)mine * (TPC / 4));
#pragma unroll
                    for (int i = 0; i < TPC / 8; i++)
                        dst[i] = make_uint4((uint32_t)col[2 * i], (uint32_t)(col[2 * i] >> 32),
                                            (uint32_t)col[2 * i + 1], (uint32_t)(col[2 * i + 1] >> 32));
                    __threadfence();
                }
            }
            pool.at += n;
        }
        if (!done && s == 0) {
            s = atomicCAS(&D.tab[idx], 0ull, tag << 40 | (mine + 1ull));
            if (s == 0) {
                id = mine;
                done = true;
            } else {
                __threadfence();   /* its column, published before the slot */
            }
        }
        if (!done) {
            bool eq = (s >> 40) == tag;
            if (eq) {
                const uint32_t o = (uint32_t)(s & kRefMask) - 1u;
                const uint4 *src = reinterpret_cast<const uint4 *>(D.cols + (uint64_t)o * (TPC / 4));
#pragma unroll
                for (int i = 0; i < TPC / 8; i++) {
                    const uint4 w = __ldcg(src + i);
                    eq &= col[2 * i] == ((uint64_t)w.y << 32 | w.x) &&
                          col[2 * i + 1] == ((uint64_t)w.w << 32 | w.z);
                }
                if (eq) {
                    id = o;
                    done = true;
                }
            }
            if (!eq) {
                idx = (idx + 1) & D.mask;
                if (++probes >= kMaxProbes) {
                    atomicOr(status, kStatusColumns);
                    done = true;
                }
            }
        }
    }
    return id;
}

/* Ids of a level's registers: eight lanes a state, a register each. */
template <int TPC>
__global__ void __launch_bounds__(kThreads)
k_state_ids(LevelDev P, IdDev D, uint32_t *status)
{
    __shared__ uint64_t sc[kWarpsPerBlock][32][TPC / 4 + 1];
    const int lane = threadIdx.x & 31, r = lane & 7;
    uint64_t *col = sc[threadIdx.x >> 5][lane];
    IdPool pool;
    const uint64_t nw = (uint64_t)gridDim.x * kWarpsPerBlock;
    for (uint64_t w = ((uint64_t)blockIdx.x * kThreads + threadIdx.x) >> 5; w * 4 < P.n; w += nw) {
        const uint64_t q = w * 4 + (lane >> 3);
        const bool want = q < P.n && r;
        uint64_t h = 0x243F6A8885A308D3ull;
        if (want) {
            const uint4 *src = reinterpret_cast<const uint4 *>(P.regs + (q * 8 + r) * TPC);
#pragma unroll
            for (int i = 0; i < TPC / 8; i++) {
                const uint4 v = src[i];
                col[2 * i] = (uint64_t)v.y << 32 | v.x;
                col[2 * i + 1] = (uint64_t)v.w << 32 | v.z;
                h = chain(chain(h, col[2 * i]), col[2 * i + 1]);
            }
        }
        const uint32_t id = intern<TPC>(D, col, h, want, pool, status, lane);
        if (q < P.n) D.ids[q * 8 + r] = r ? id : (uint32_t)P.task[q] << 8 | P.live[q];
    }
}

/* Exact compare of child A (class jA of the warp's parent written to rdA; its
   column and flags in shared memory) with child B (parent qB of the level in
   HBM + micro-op uB), the whole warp cooperating: lane t rebuilds test t of
   child B (every register, the flags) and __all_sync decides. The requesting
   lane has already checked the task and (when it is part of the key) the live
   mask. All lanes must call it. Used where a level's column ids do not fit. */
template <int TPC>
__device__ bool warp_child_equal(const LevelDev &P, const InsertState<TPC> &A, int T, int jA,
                                 uint32_t rdA, uint64_t qB, uint32_t uB, int lane)
{
    bool ok = true;
    if (lane < T) {
        const uint32_t rdB = UOP_RD(uB);
        const uint32_t resA = reinterpret_cast<const uint16_t *>(A.colA[jA])[lane];
        const uint4 f = A.flagsA[jA];
        const uint32_t b = plane_bit<TPC>(lane);
        const uint32_t fA = (f.x >> b & 1u) | (f.y >> b & 1u) << 1 | (f.z >> b & 1u) << 2 |
                            (f.w >> b & 1u) << 3;
        const uint16_t *RB = P.regs + qB * 8 * TPC + lane;
        const uint32_t a2 = RB[UOP_A(uB) * TPC], b2 = RB[UOP_B(uB) * TPC];
        const uint32_t resB = pca_alu(UOP_OP(uB), a2, b2, UOP_IMM(uB));
        const uint32_t fB = pca_alu_flags(UOP_OP(uB), a2, b2, UOP_IMM(uB), resB,
                                          P.flags[qB * TPC + lane]);
        ok = fA == fB;
#pragma unroll
        for (uint32_t r = 1; r < 8; r++) {
            const uint32_t vA = r == rdA ? resA
                                         : (uint32_t)reinterpret_cast<const uint16_t *>(A.R[r])[lane];
            const uint32_t vB = r == rdB ? resB : (uint32_t)RB[r * TPC];
            ok &= vA == vB;
        }
    }
    return __all_sync(0xFFFFFFFFu, ok);
}

/* A child's new column and flags depend on its value class alone, not on the
   destination, so a warp forms the values of its parent's classes, a class a
   lane, in runs of one op, gives their columns exact ids, and then takes the
   run's children (class, destination) that may be a representative, 32 at a
   time. IDS: two children are compared by ids; else, on a level whose ids do
   not fit, column by column (warp_child_equal).

   Bound: memory latency (45% issue; a tag match is four dependent loads) with
   32 warps an SM, 64 registers a thread: five CTAs of 48 registers spill and
   measured 4% slower. Level 3 of a 32-test search (24,547 parents, 15.5M
   children, 7.9M of them looked up, 5.3M kept): hashing each child's column
   and comparing columns by the warp took 943M warp instructions, 1.40 ms;
   hashing by class 695M, 1.16 ms; with ids 311M, 0.61 ms (0.75 with the
   ids of the level's registers and the clearing of their table).

   The child bitmap is kept beside the table: a child that takes a slot
   toggles its bit, and one that takes it from a later sibling the other's
   too, so that in whatever order the toggles land each slot's last holder has
   its bit set and nobody else (a scan of the 256 MB table for its holders
   took 0.09 ms of the level and a launch, the toggles 0.06). */
__device__ __forceinline__ void toggle_child(uint32_t *bitmap, uint64_t child)
{
    atomicXor(&bitmap[child >> 5], 1u << (child & 31));
}

template <int TPC, bool IDS>
__global__ void __launch_bounds__(kThreads, 4)
k_expand_insert(LevelDev P, TaskDev task, unsigned long long *table, uint64_t tmask,
                uint32_t *status, uint32_t split_log2, const uint32_t *fcr_up, uint32_t *next, IdDev D,
                uint32_t *bitmap)
{
    __shared__ InsertState<TPC> sws[kWarpsPerBlock];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    InsertState<TPC> &ws = sws[wib];
    const uint32_t split = 1u << split_log2;
    /* a work item is a parent (split 1) or one of `split` slices of its
       chunk list: small levels spread each parent over several warps. Warps
       draw items from a counter (`next`, zero at launch; lane 0 fetches the
       next item while the warp works on the current one): a parent's cost
       (its children, their probes and exact compares) varies widely, and
       fixed shares left the first SMs idle for ~18% of the launch while the
       last finished (a warp stages its own parent, so no L1 sharing is lost;
       measured 1.59 -> 1.48 ms per solve). Items < 2^33 (levels below 2^28
       states, slices only for levels below 2^12). */
    const uint64_t items = P.n << split_log2;
    IdPool pool;
    uint32_t nx = 0;
    if (lane == 0) nx = atomicAdd(next, 1u);
    for (uint64_t it = __shfl_sync(0xFFFFFFFFu, nx, 0); it < items;
         it = __shfl_sync(0xFFFFFFFFu, nx, 0)) {
        if (lane == 0) nx = atomicAdd(next, 1u);
        const uint64_t q = it >> split_log2;
        const uint32_t g = (uint32_t)it & (split - 1);
        const uint32_t tid = P.task[q];
        if (!task.active[tid]) continue;
        const int T = task.T[tid];
        __syncwarp();
        if (lane < TPC) {
            const uint4 w = reinterpret_cast<const uint4 *>(P.regs + q * 8 * TPC)[lane];
            uint32_t *row = &ws.R[lane / (TPC / 8)][lane % (TPC / 8) * 4];
            row[0] = w.x; row[1] = w.y; row[2] = w.z; row[3] = w.w;
            ws.F[lane] = P.flags[q * TPC + lane];
        }
        if (IDS && lane < 8) ws.ids[lane] = D.ids[q * 8 + lane];
        const uint32_t live = P.live[q];
        const uint64_t first_child = P.child_off[q];
        __syncwarp();
        if (lane >= 1 && lane < 8) ws.colh[lane] = col_final(lane, hash_column<TPC>(ws.R[lane]));
        if (lane >= 8 && lane < 12) {   /* the parent's flags, a plane a lane */
            uint32_t x = 0;
            for (int t = 0; t < TPC; t += 2)
                x = x * 2 + (ws.F[t] >> (lane - 8) & 1u) + ((ws.F[t + 1] >> (lane - 8) & 1u) << 16);
            reinterpret_cast<uint32_t *>(&ws.flagsA[32])[lane - 8] = x;
        }
        __syncwarp();
        uint64_t regsum = task_final(tid);
#pragma unroll
        for (int r = 1; r < 8; r++) regsum += ws.colh[r];
        const uint32_t m = (live >> 1) & 127u;
        const uint32_t v0 = c_vc_off[m];
        const uint32_t k0 = c_vchunk_off[m], k1 = c_vchunk_off[m + 1];
        const uint32_t per = (k1 - k0 + split - 1) >> split_log2;
        const uint32_t ka = min(k1, k0 + g * per), kb = min(k1, ka + per);
        const uint32_t wdead = deadable_writes(P, fcr_up, q);
        const uint32_t wldi = fcr_up && (P.own[q] & 1u) ? P.rdl[q] : 0u;
        const bool twin_later = P.twin[q] != 0;
        for (uint32_t k = ka; k < kb; k++) {
            const uint32_t ch = c_vchunks[k], start = ch >> 8, cnt = ch & 255u;
            const uint32_t uv = c_vc_uop[v0 + start + min((uint32_t)lane, cnt - 1)];
            const uint32_t op = UOP_OP(uv);
            if (twin_later && op != PCA_OP_LDI) continue;   /* k_twins */
            /* the children that may be a representative (c_kid leaves out
               the same-state duplicates of an earlier sibling) */
            uint32_t nk = 0;
            __syncwarp();   /* the previous chunk's children are done */
            for (uint32_t i0 = 0; i0 < cnt * 8; i0 += 32) {
                const uint32_t i = i0 + lane, rd = i & 7u;
                const uint32_t u = __shfl_sync(0xFFFFFFFFu, uv, (int)(i >> 3) & 31);
                bool valid = i < cnt * 8 && c_kid[(v0 + start) * 8 + i] != 0xFFFFu;
                const bool reads_rd = uop_reads(u, rd);
                if ((wdead >> rd & 1u) && op != PCA_OP_LDI && !reads_rd) valid = false;
                if (ldi_swap((u & ~(7u << 5)) | rd << 5, wldi)) valid = false;
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, valid);
                if (valid) ws.kids[nk + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)i;
                nk += __popc(bal);
            }
            if (!nk) continue;
            {
                uint64_t h, hf;
                class_values_any<TPC>(op, ws, UOP_A(uv), UOP_B(uv), UOP_IMM(uv), T, lane, h, hf);
                ws.hA[lane] = h;
                ws.hfA[lane] = hf;
                if (IDS) {
                    const bool mine = (uint32_t)lane < cnt;
                    const uint32_t id = intern<TPC>(D, ws.colA[lane], h, mine, pool, status, lane);
                    ws.idA[lane] = id;
                    if (mine) {
                        const uint64_t at = q * D.stride + start + lane;
                        D.cls_id[at] = id;
                        D.cls_flags[at] = ws.flagsA[lane];
                    }
                    __threadfence();   /* before any slot names these classes */
                }
            }
            __syncwarp();
            for (uint32_t i0 = 0; i0 < nk; i0 += 32) {
            const bool valid = i0 + lane < nk;
            const uint32_t kid = ws.kids[valid ? i0 + lane : 0];
            const uint32_t cls = kid >> 3, rd = kid & 7u;
            const uint32_t c = c_kid[(v0 + start) * 8 + kid];
            uint64_t H = regsum - ws.colh[rd] + col_final(rd, ws.hA[cls]) + ws.hfA[cls];
            if (task.key_live) H += live_final(live | (1u << rd));
            const uint64_t ref = (q << 12) | c;
            const unsigned long long mine = ((H >> 40) << 40) | (ref + 1);
            uint64_t idx = H & tmask;
            uint32_t probes = 0;
            bool done = !valid;
            /* lanes probe in parallel; a tag match is settled by an exact
               warp-wide compare, one requesting lane at a time */
            while (__any_sync(0xFFFFFFFFu, !done)) {
                bool needcmp = false;
                unsigned long long s = 0;
                if (!done) {
                    s = IDS ? load_acquire(&table[idx])
                            : *((volatile unsigned long long *)&table[idx]);
                    if (s == 0) {
                        const unsigned long long old = atomicCAS(&table[idx], 0ull, mine);
                        if (old == 0) {
                            toggle_child(bitmap, first_child + c);
                            done = true;
                        } else {
                            s = old;
                            if (IDS) __threadfence();   /* as after an acquiring load */
                        }
                    }
                    if (!done) needcmp = (s >> 40) == (mine >> 40);
                }
                /* a tag match first settles the stored child's task, live
                   mask and micro-op in its own lane (all lanes at once) */
                uint64_t qB = 0;
                uint32_t uB = 0, cB = 0;
                uint4 b0 = make_uint4(0, 0, 0, 0), b1 = b0;   /* the parent's ids */
                if (needcmp) {
                    const uint64_t oref = (s & kRefMask) - 1;
                    qB = oref >> 12;
                    uint32_t liveB = live, tB = tid;
                    if (IDS) {
                        const uint4 *src = reinterpret_cast<const uint4 *>(D.ids + qB * 8);
                        b0 = src[0];
                        b1 = src[1];
                        liveB = b0.x & 0xFFu;
                        tB = b0.x >> 8;
                    } else if (qB != q) {
                        tB = P.task[qB];
                        liveB = P.live[qB];
                    }
                    needcmp = tB == tid;
                    const uint2 k = c_cand_k[c_cand_off_g[(liveB >> 1) & 127u] + (uint32_t)(oref & 4095)];
                    uB = k.x;
                    cB = k.y;
                    if (task.key_live && (live | (1u << rd)) != (liveB | (1u << UOP_RD(uB))))
                        needcmp = false;
                }
                bool eq = false;
                if (IDS) {
                    if (needcmp) {
                        const uint64_t at = qB * D.stride + cB;
                        const uint32_t idB = __ldcg(D.cls_id + at);
                        const uint4 fB = __ldcg(D.cls_flags + at), fA = ws.flagsA[cls];
                        const uint32_t B[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
                        const uint32_t idA = ws.idA[cls], rdB = UOP_RD(uB);
                        eq = fA.x == fB.x && fA.y == fB.y && fA.z == fB.z && fA.w == fB.w;
#pragma unroll
                        for (uint32_t r = 1; r < 8; r++)
                            eq &= (r == rd ? idA : ws.ids[r]) == (r == rdB ? idB : B[r]);
                    }
                } else {
                    uint32_t req = __ballot_sync(0xFFFFFFFFu, needcmp);
                    while (req) {
                        const int j = __ffs(req) - 1;
                        req &= req - 1;
                        const uint32_t kj = __shfl_sync(0xFFFFFFFFu, kid, j);
                        const uint32_t ubj = __shfl_sync(0xFFFFFFFFu, uB, j);
                        const uint64_t qbj = __shfl_sync(0xFFFFFFFFu, qB, j);
                        const bool e = warp_child_equal<TPC>(P, ws, T, (int)(kj >> 3), kj & 7u, qbj,
                                                             ubj, lane);
                        if (lane == j) eq = e;
                    }
                }
                if (!done) {
                    if (needcmp && eq) {
                        /* same state: keep the smaller ref (the DFS-first child) */
                        uint64_t oref = (s & kRefMask) - 1;
                        while (ref < oref) {
                            const unsigned long long old = atomicCAS(&table[idx], s, mine);
                            if (old == s) {
                                toggle_child(bitmap, first_child + c);
                                toggle_child(bitmap, P.child_off[oref >> 12] + (oref & 4095));
                                break;
                            }
                            s = old;
                            oref = (s & kRefMask) - 1;
                        }
                        done = true;
                    } else {
                        idx = (idx + 1) & tmask;
                        if (++probes >= kMaxProbes) {
                            atomicOr(status, kStatusTableFull);
                            done = true;
                        }
                    }
                }
            }
            }
        }
    }
}

/* Flag twins. Two states of a level with the same registers, live mask and
   task but different flags (e.g. two independent instructions in either
   order, or two ops that write the same value with different flags) have,
   for every flag-setting candidate c (every op but LDI), children that are
   the same state under either pruning key: the same registers, c's flags
   and the same live mask; and c has the same index in both parents' lists
   (the lists depend on live only). The earlier state's child is the smaller
   ref, so no flag-setting child of a later twin is ever the DFS-first
   representative: k_twins marks the later twins (twin[q] = 1) and the insert
   kernel skips those children. One warp per state (lane = test): a hash of
   r1..r7, live and task, then an open-addressed table whose slot keeps the
   class's lowest rank, every tag match settled by an exact warp-wide
   compare. Probing is bounded (kStatusTableFull). twin[] is zeroed
   beforehand. */
template <int TPC>
__global__ void k_twins(LevelDev P, TaskDev task, unsigned long long *table, uint64_t tmask,
                        uint8_t *twin, uint32_t *status)
{
    const int lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t q = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < P.n; q += nw) {
        const uint32_t tid = P.task[q];
        if (!task.active[tid]) continue;
        const uint32_t live = P.live[q];
        uint32_t col[7];
        uint64_t h = 0;
        if (lane < TPC) {
            const uint16_t *src = P.regs + q * 8 * TPC + lane;
            uint64_t w = 0x243F6A8885A308D3ull ^ (uint64_t)lane;
#pragma unroll
            for (int r = 1; r < 8; r++) {
                col[r - 1] = src[r * TPC];
                w = chain(w, col[r - 1]);
            }
            h = fmix64(w);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) h += __shfl_xor_sync(0xFFFFFFFFu, h, o);
        const uint64_t H = h + live_final(live) + task_final(tid);
        const unsigned long long mine = ((H >> 40) << 40) | (q + 1);
        uint64_t idx = H & tmask;
        uint32_t probes = 0;
        for (;;) {
            unsigned long long s = 0;
            if (lane == 0) {
                s = *((volatile unsigned long long *)&table[idx]);
                if (s == 0) s = atomicCAS(&table[idx], 0ull, mine);
            }
            s = __shfl_sync(0xFFFFFFFFu, s, 0);
            if (s == 0) break;   /* the first of its class so far */
            bool eq = false;
            if ((s >> 40) == (mine >> 40)) {
                const uint64_t qB = (s & kRefMask) - 1;
                eq = P.task[qB] == tid && P.live[qB] == live;
                if (eq) {
                    bool ok = true;
                    if (lane < TPC) {
                        const uint16_t *srcB = P.regs + qB * 8 * TPC + lane;
#pragma unroll
                        for (int r = 1; r < 8; r++) ok &= srcB[r * TPC] == col[r - 1];
                    }
                    eq = __all_sync(0xFFFFFFFFu, ok);
                }
            }
            if (eq) {
                /* one class: the slot keeps the lowest rank, every other
                   member is marked */
                if (lane == 0) {
                    unsigned long long cur = s;
                    for (;;) {
                        const uint64_t m = (cur & kRefMask) - 1;
                        if (q > m) { twin[q] = 1; break; }
                        const unsigned long long old = atomicCAS(&table[idx], cur, mine);
                        if (old == cur) { twin[m] = 1; break; }
                        cur = old;
                    }
                }
                break;
            }
            idx = (idx + 1) & tmask;
            if (++probes >= kMaxProbes) {
                if (lane == 0) atomicOr(status, kStatusTableFull);
                break;
            }
        }
    }
}

/* Keep every child (no pruning): set all bits below `total`. */
__global__ void k_mark_all(uint32_t *bitmap, uint64_t words, uint64_t total)
{
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < words;
         w += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t lo = w * 32;
        uint32_t v = 0xFFFFFFFFu;
        if (lo + 32 > total) v = total > lo ? (uint32_t)((1ull << (total - lo)) - 1) : 0u;
        bitmap[w] = v;
    }
}

__global__ void k_popc(const uint32_t *bitmap, uint64_t words, uint64_t *cnt)
{
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < words;
         w += (uint64_t)gridDim.x * blockDim.x)
        cnt[w] = __popc(bitmap[w]);
}

/* child_off[i] = number of candidates of state i, 0 when its task is not
   searched any more (scanned afterwards). */
__global__ void k_child_counts(const uint8_t *live, const uint16_t *task, const uint8_t *active,
                               uint64_t n, uint64_t *cnt)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t m = (live[i] >> 1) & 127u;
        cnt[i] = active[task[i]] ? c_cand_off[m + 1] - c_cand_off[m] : 0;
    }
}

/* ---- the bookkeeping of a small level -----------------------------------------
   A level of a few hundred states is built in launches of a few microseconds
   each, so their number is its time: what has to be cleared is cleared by one
   launch (nine to ten memsets), and counts are formed and scanned by one block
   (a counting launch, two to four of the scan and a memset). A solve that
   builds two such levels takes 493 us where it took 574. */
constexpr int kClearMax = 10;
struct ClearList {
    void *p[kClearMax];          /* 16-byte aligned */
    uint64_t bytes[kClearMax];
    uint32_t value[kClearMax];   /* 0 or ~0 */
    int n;
    void add(void *at, uint64_t count, uint32_t v = 0)
    {
        p[n] = at;
        bytes[n] = count;
        value[n++] = v;
    }
};

__global__ void k_clear(const __grid_constant__ ClearList L)
{
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int r = 0; r < L.n; r++) {
        const uint32_t v = L.value[r];
        for (uint64_t i = t; i < L.bytes[r] / 16; i += (uint64_t)gridDim.x * blockDim.x)
            reinterpret_cast<uint4 *>(L.p[r])[i] = make_uint4(v, v, v, v);
        const uint64_t tail = L.bytes[r] % 16;
        if (t < tail) reinterpret_cast<uint8_t *>(L.p[r])[L.bytes[r] - tail + t] = (uint8_t)v;
    }
}

/* The exclusive offsets of a block's counts, four a thread (1,024 threads),
   and their sum in every thread. */
__device__ __forceinline__ uint32_t block_offsets(const uint32_t (&v)[4], uint32_t (&off)[4],
                                                  uint32_t (&sums)[33])
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t s = v[0] + v[1] + v[2] + v[3], inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += x;
    }
    if (lane == 31) sums[w] = inc;
    __syncthreads();
    if (w == 0) {
        const uint32_t own = sums[lane];
        uint32_t all = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, all, o);
            if (lane >= o) all += x;
        }
        sums[lane] = all - own;
        if (lane == 31) sums[32] = all;
    }
    __syncthreads();
    uint32_t run = sums[w] + inc - s;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        off[k] = run;
        run += v[k];
    }
    const uint32_t total = sums[32];
    __syncthreads();
    return total;
}

/* child_off[0..n] of a level of at most kSmallParents states, one block. */
constexpr uint64_t kSmallParents = 16384;
__global__ void __launch_bounds__(1024) k_child_offsets(const uint8_t *live, const uint16_t *task,
                                                       const uint8_t *active, uint64_t n,
                                                       uint64_t *child_off)
{
    __shared__ uint32_t sums[33];
    uint64_t carry = 0;
    for (uint64_t base = 0; base < n; base += 4096) {
        const uint64_t i = base + threadIdx.x * 4;
        uint32_t v[4], off[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = 0;
            if (i + k < n && active[task[i + k]]) {
                const uint32_t m = (live[i + k] >> 1) & 127u;
                v[k] = c_cand_off[m + 1] - c_cand_off[m];
            }
        }
        const uint32_t total = block_offsets(v, off, sums);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (i + k < n) child_off[i + k] = carry + off[k];
        carry += total;
    }
    if (threadIdx.x == 0) child_off[n] = carry;
}

/* The ranks of a bitmap of at most kSmallWords words, word_off[0..words],
   and the number of set bits, one block. */
constexpr uint64_t kSmallWords = 32768;
__global__ void __launch_bounds__(1024) k_word_offsets(const uint32_t *bitmap, uint64_t words,
                                                      uint64_t *word_off, unsigned long long *total)
{
    __shared__ uint32_t sums[33];
    uint64_t carry = 0;
    for (uint64_t base = 0; base < words; base += 4096) {
        const uint64_t i = base + threadIdx.x * 4;
        uint32_t v[4], off[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = i + k < words ? __popc(bitmap[i + k]) : 0;
        const uint32_t sum = block_offsets(v, off, sums);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (i + k < words) word_off[i + k] = carry + off[k];
        carry += sum;
    }
    if (threadIdx.x == 0) {
        word_off[words] = carry;
        *total = carry;
    }
}

/* One warp's shared memory in the materialisation: the parent's register
   block in the level's own layout (8 columns of TPC tests) and the current
   child's new column and flags, from which each lane writes one 16-byte
   piece of the child. */
template <int TPC>
struct MatState {
    __align__(16) uint16_t PR[8 * TPC];
    __align__(16) uint16_t CB[32];   /* 32 / TPC children at a time */
    __align__(16) uint8_t FB[32];
};

/* Write the marked children of each parent, in rank (DFS) order, by TPC lanes
   each (with 16 tests two children at a time: level 3 of an 11-test search,
   5.3M states, 0.62 -> 0.48 ms). A child's register block (8 x TPC halves) is
   written as TPC 16-byte pieces, one per lane, and its flags as TPC/16
   pieces: lane t first computes the new value
   and flags of test t into shared memory, then lane L copies piece L from
   the parent's block, or from the new column when the piece lies in the
   written register's column. Level blocks start on 256-byte boundaries (the
   arena's allocation unit) and a state's block is 256 or 512 bytes, so
   every piece is 16-byte aligned. */
template <int TPC>
__global__ void __launch_bounds__(kThreads)
k_materialize(LevelDev P, TaskDev task, const uint32_t *bitmap, const uint64_t *word_off,
              LevelOut C, uint32_t split_log2, uint32_t *fcr, const uint32_t *fcr_up)
{
    static_assert(TPC == 16 || TPC == 32, "a state holds 16 or 32 tests");
    constexpr int kPieces = 8 * TPC * 2 / 16;   /* = TPC: a piece a lane of the group */
    constexpr int kFlagPieces = TPC / 16;
    constexpr int kPiecesPerCol = TPC / 8;
    __shared__ MatState<TPC> sms[kWarpsPerBlock];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int t = lane % TPC, grp = lane / TPC;   /* test (and piece), child of the pair */
    MatState<TPC> &ms = sms[wib];
    const uint32_t my_col = (uint32_t)t / kPiecesPerCol;   /* column of piece t */
    const uint4 *my_new = reinterpret_cast<const uint4 *>(ms.CB + grp * TPC) + t % kPiecesPerCol;
    const uint4 *my_old = reinterpret_cast<const uint4 *>(ms.PR) + t;
    const uint64_t nw = (uint64_t)gridDim.x * kWarpsPerBlock;
    const uint32_t split = 1u << split_log2;
    /* work items as in k_expand_insert: a parent, or a slice of its
       32-candidate groups */
    for (uint64_t it = (uint64_t)blockIdx.x * kWarpsPerBlock + wib; it < (P.n << split_log2);
         it += nw) {
        const uint64_t q = it >> split_log2;
        const uint32_t g = (uint32_t)it & (split - 1);
        const uint32_t tid = P.task[q];
        if (!task.active[tid]) continue;
        const int T = task.T[tid];
        __syncwarp();
        if (lane < kPieces)
            reinterpret_cast<uint4 *>(ms.PR)[lane] =
                reinterpret_cast<const uint4 *>(P.regs + q * 8 * TPC)[lane];
        const uint32_t pf = P.flags[q * TPC + t];
        const uint32_t live = P.live[q];
        __syncwarp();
        const uint32_t m = (live >> 1) & 127u;
        const uint32_t base = c_cand_off[m], nc = c_cand_off[m + 1] - base;
        const uint64_t off = P.child_off[q];
        const uint32_t W = deadable_writes(P, fcr_up, q);
        const uint32_t groups = (nc + 31) >> 5;
        const uint32_t per = (groups + split - 1) >> split_log2;
        const uint32_t ga = min(groups, g * per), gb = min(groups, ga + per);
        for (uint32_t c0 = ga * 32; c0 < gb * 32; c0 += 32) {
            /* each lane settles its own candidate (kept?, rank, micro-op and
               the child's links) so the per-child loop below needs no
               global load */
            const uint32_t c = c0 + lane;
            bool keep = false;
            uint64_t rank = 0;
            uint32_t u = 0;
            if (c < nc) {
                const uint64_t L = off + c;
                const uint32_t wv = bitmap[L >> 5];
                keep = (wv >> (L & 31)) & 1u;
                if (keep) {
                    rank = word_off[L >> 5] + __popc(wv & ((1u << (L & 31)) - 1u));
                    u = c_cand_uop[base + c];
                    C.live[rank] = (uint8_t)(live | (1u << UOP_RD(u)));
                    C.rdl[rank] = (uint8_t)UOP_RD(u);
                    C.task[rank] = (uint16_t)tid;
                    C.parent[rank] = (uint32_t)q;
                    C.cidx[rank] = (uint16_t)c;
                    /* a write read by u is used; the one u overwrites is gone */
                    C.own[rank] = (uint8_t)((W & ~((1u << UOP_A(u)) | (1u << UOP_B(u)) |
                                                   (1u << UOP_RD(u))) & 0xFEu) |
                                            (UOP_OP(u) == PCA_OP_LDI ? 1u : 0u));
                    /* first kept child of q per written register */
                    if (fcr) atomicMin(&fcr[q * 8 + UOP_RD(u)], (uint32_t)rank);
                }
            }
            uint32_t bal = __ballot_sync(0xFFFFFFFFu, keep);
            while (bal) {
                /* this lane group's child: the first set bit, or the second */
                uint32_t mine = bal;
                bal &= bal - 1;
                if (TPC == 16) {
                    mine = grp ? bal : mine;
                    bal &= bal - 1;
                }
                const int j = __ffs((int)mine) - 1;
                const uint64_t rk = __shfl_sync(0xFFFFFFFFu, rank, j < 0 ? 0 : j);
                const uint32_t uj = __shfl_sync(0xFFFFFFFFu, u, j < 0 ? 0 : j);
                const uint32_t op = UOP_OP(uj), rd = UOP_RD(uj);
                {
                    const uint32_t a = ms.PR[UOP_A(uj) * TPC + t];
                    const uint32_t b = ms.PR[UOP_B(uj) * TPC + t];
                    uint32_t res = pca_alu(op, a, b, UOP_IMM(uj));
                    uint32_t f = pca_alu_flags(op, a, b, UOP_IMM(uj), res, pf);
                    if (t >= T) { res = 0; f = 0; }
                    ms.CB[lane] = (uint16_t)res;
                    ms.FB[lane] = (uint8_t)f;
                }
                __syncwarp();
                if (j >= 0) {
                    const uint4 pv = *(my_col == rd ? my_new : my_old);
                    reinterpret_cast<uint4 *>(C.regs + rk * 8 * TPC)[t] = pv;
                    /* the lane holding tests 0..7 of a column also writes
                       tests 0..3 of it into the probe (8 lanes, 64 bytes) */
                    if (t % kPiecesPerCol == 0)
                        reinterpret_cast<uint2 *>(C.probe + rk * 32)[my_col] = make_uint2(pv.x, pv.y);
                    if (t < kFlagPieces)
                        reinterpret_cast<uint4 *>(C.flags + rk * TPC)[t] =
                            reinterpret_cast<const uint4 *>(ms.FB + grp * TPC)[t];
                }
                __syncwarp();
            }
        }
    }
}

/* The lean form of k_materialize, for a level that only the last position
 * reads (the lane-per-prefix scan: each state's 64-byte probe, its links,
 * and on a hit the registers that k_suffix_lanes recomputes from the
 * parent). Per kept child it writes live, rdl, task, parent, cidx, own and
 * the probe, computed from the parent's probe: no register block and no
 * flags, 64 bytes a state instead of 8 x TPC x 2 + TPC + 64. A warp takes a
 * parent (or a slice of its 32-candidate groups, as k_materialize), stages
 * the parent's probe in shared memory, and each lane settles its own
 * candidate. */
template <int TPC>
__global__ void __launch_bounds__(kThreads)
k_materialize_probe(LevelDev P, TaskDev task, const uint32_t *bitmap, const uint64_t *word_off,
                    LevelOut C, uint32_t split_log2, const uint32_t *fcr_up, uint32_t *next)
{
    static_assert(TPC == 16 || TPC == 32, "a state holds 16 or 32 tests");
    __shared__ __align__(16) uint16_t spp[kWarpsPerBlock][8][4];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    uint16_t (&PP)[8][4] = spp[wib];
    const uint32_t split = 1u << split_log2;
    /* work items drawn from a counter, as in k_expand_insert (measured
       0.03 ms faster per solve than fixed shares) */
    const uint64_t items = P.n << split_log2;
    uint32_t nx = 0;
    if (lane == 0) nx = atomicAdd(next, 1u);
    for (uint64_t it = __shfl_sync(0xFFFFFFFFu, nx, 0); it < items;
         it = __shfl_sync(0xFFFFFFFFu, nx, 0)) {
        if (lane == 0) nx = atomicAdd(next, 1u);
        const uint64_t q = it >> split_log2;
        const uint32_t g = (uint32_t)it & (split - 1);
        const uint32_t tid = P.task[q];
        if (!task.active[tid]) continue;
        const int T = task.T[tid];
        __syncwarp();
        if (lane < 8)
            reinterpret_cast<uint2 *>(&PP[0][0])[lane] =
                reinterpret_cast<const uint2 *>(P.probe + q * 32)[lane];
        const uint32_t live = P.live[q];
        __syncwarp();
        const uint32_t m = (live >> 1) & 127u;
        const uint32_t base = c_cand_off[m], nc = c_cand_off[m + 1] - base;
        const uint64_t off = P.child_off[q];
        const uint32_t W = deadable_writes(P, fcr_up, q);
        const uint32_t groups = (nc + 31) >> 5;
        const uint32_t per = (groups + split - 1) >> split_log2;
        const uint32_t ga = min(groups, g * per), gb = min(groups, ga + per);
        for (uint32_t c = ga * 32 + lane; c < gb * 32; c += 32) {
            if (c >= nc) continue;
            const uint64_t L = off + c;
            const uint32_t wv = bitmap[L >> 5];
            if (!((wv >> (L & 31)) & 1u)) continue;
            const uint64_t rank = word_off[L >> 5] + __popc(wv & ((1u << (L & 31)) - 1u));
            const uint32_t u = c_cand_uop[base + c];
            const uint32_t rd = UOP_RD(u), ra = UOP_A(u), rb = UOP_B(u);
            C.live[rank] = (uint8_t)(live | (1u << rd));
            C.rdl[rank] = (uint8_t)rd;
            C.task[rank] = (uint16_t)tid;
            C.parent[rank] = (uint32_t)q;
            C.cidx[rank] = (uint16_t)c;
            C.own[rank] = (uint8_t)((W & ~((1u << ra) | (1u << rb) | (1u << rd)) & 0xFEu) |
                                    (UOP_OP(u) == PCA_OP_LDI ? 1u : 0u));
            /* the written register on tests 0..3 (0 past the task's tests,
               as k_materialize writes them) */
            uint32_t nv[4];
#pragma unroll
            for (int t = 0; t < 4; t++)
                nv[t] = t < T ? pca_alu(UOP_OP(u), PP[ra][t], PP[rb][t], UOP_IMM(u)) & 0xFFFFu
                              : 0u;
            const uint32_t lo = nv[0] | (nv[1] << 16), hi = nv[2] | (nv[3] << 16);
            uint4 *dst = reinterpret_cast<uint4 *>(C.probe + rank * 32);
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const uint4 old = reinterpret_cast<const uint4 *>(&PP[0][0])[h];
                uint4 v = old;
                if (rd == 2u * h) { v.x = lo; v.y = hi; }
                if (rd == 2u * h + 1) { v.z = lo; v.w = hi; }
                dst[h] = v;
            }
        }
    }
}

/* hist[task][mask] += states of that task with that liveness mask. Lanes
   with the same key are counted by one atomic (states of a level are
   grouped by task and mostly by mask). With n_dev set, the level holds
   min(n, *n_dev) states (n is then the space written, an upper bound). */
__global__ void k_task_hist(const uint8_t *live, const uint16_t *task, uint64_t n,
                            const unsigned long long *n_dev, unsigned long long *hist)
{
    if (n_dev && *n_dev < n) n = *n_dev;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t n_round = (n + 31) & ~31ull;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_round; i += stride) {
        const bool valid = i < n;
        const uint32_t key = valid ? (uint32_t)task[i] * 128u + ((live[i] >> 1) & 127u) : ~0u;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
        if (valid && (threadIdx.x & 31) == __ffs(peers) - 1)
            atomicAdd(&hist[key], (unsigned long long)__popc(peers));
    }
}

/* The same with a per-block histogram in shared memory (nbins u32 counters,
   nbins = tasks x 128 <= 4096), flushed with one global atomic per nonzero
   bin: a level's states crowd a few bins, and per-warp global atomics on
   them serialize. */
__global__ void k_task_hist_smem(const uint8_t *live, const uint16_t *task, uint64_t n,
                                 const unsigned long long *n_dev, uint32_t nbins,
                                 unsigned long long *hist)
{
    extern __shared__ uint32_t sh_hist[];
    if (n_dev && *n_dev < n) n = *n_dev;
    for (uint32_t b = threadIdx.x; b < nbins; b += blockDim.x) sh_hist[b] = 0;
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t n_round = (n + 31) & ~31ull;
    /* four states a thread in flight: one at a time, 5.3M states took 46 us,
       waiting for their bytes; 22 so */
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n_round;
         i0 += 4 * stride) {
        uint32_t key[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint64_t i = i0 + k * stride;
            key[k] = i < n ? (uint32_t)task[i] * 128u + ((live[i] >> 1) & 127u) : ~0u;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key[k]);
            if ((threadIdx.x & 31) == __ffs(peers) - 1 && key[k] < nbins)
                atomicAdd(&sh_hist[key[k]], (uint32_t)__popc(peers));
        }
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < nbins; b += blockDim.x)
        if (sh_hist[b]) atomicAdd(&hist[b], (unsigned long long)sh_hist[b]);
}

/* ---- solutions ----------------------------------------------------------- */

struct SolBuf {
    unsigned long long *count;    /* solving (prefix, mids, class) records */
    ulonglong2 *rec;              /* x = prefix rank, y = m1<<32 | m2<<16 | class */
    uint64_t cap;
    ulonglong2 *firsts;           /* first-only stages, in place of the records: per task the
                                     smallest packed DFS-order key (x) and the programs of its
                                     records less one (y; both start as all ones) */
    const uint16_t *task;         /* task of each prefix (with firsts) */
    unsigned long long *evals;    /* value-class evaluations the suffix kernels ran
                                     (each class of an operand pair counts one) */
};

/* Adds a warp's per-lane evaluation counts to S.evals (all lanes call it). */
__device__ __forceinline__ void flush_evals(const SolBuf &S, unsigned long long nev, int lane)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) nev += __shfl_down_sync(0xFFFFFFFFu, nev, o);
    if (lane == 0 && nev) atomicAdd(S.evals, nev);
}

/* A solving record: prefix q, middles m1, m2, value class vc, whose first
   candidate in DFS order is first_c and which has n of them. */
__device__ __forceinline__ void record(const SolBuf &S, uint64_t q, uint32_t m1, uint32_t m2,
                                       uint32_t vc, uint32_t first_c, uint32_t n)
{
    const unsigned long long slot = atomicAdd(S.count, 1ull);
    if (S.firsts) {
        ulonglong2 *f = S.firsts + S.task[q];
        atomicMin(&f->x, ((unsigned long long)(q & 0xFFFFFFFull) << 36) |
                             ((unsigned long long)m1 << 24) | ((unsigned long long)m2 << 12) |
                             first_c);
        atomicAdd(&f->y, (unsigned long long)n);
    } else if (slot < S.cap) {
        S.rec[slot] = make_ulonglong2(q, ((unsigned long long)m1 << 32) | (m2 << 16) | vc);
    }
}

/* The same by a class of mask m (index vc in its list). */
__device__ __forceinline__ void record_solution(const SolBuf &S, uint64_t q, uint32_t m1,
                                                uint32_t m2, uint32_t vc, uint32_t m)
{
    const uint32_t i = c_vc_off[m] + vc;
    record(S, q, m1, m2, vc, c_vc_first[i], c_vc_n[i]);
}

/* Leaf check of a materialized level (count mode): state q solves through
 * live register r when regs[q][r][t] == target[t] for every test. */
template <int TPC>
__global__ void k_leaf(LevelDev P, TaskDev task, SolBuf S)
{
    const int lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t q = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < P.n; q += nw) {
        const uint32_t tid = P.task[q];
        if (!task.active[tid]) continue;
        const int T = task.T[tid];
        const uint32_t tgt = lane < T ? task.target[tid * 32 + lane] : 0u;
        const uint32_t live = P.live[q];
        for (uint32_t r = 1; r < 8; r++) {
            if (!((live >> r) & 1u)) continue;
            bool ok = lane >= T || P.regs[q * 8 * TPC + r * TPC + lane] == tgt;
            if (__all_sync(0xFFFFFFFFu, ok) && lane == 0) record(S, q, 0, 0, r, r, 1);
        }
    }
}

/* The leaf check past depth 1. At depth K - 1 no state held the target in a
 * live register (its leaf check found nothing), so a state of level K can
 * hold it only in the register its last instruction wrote. A lane per state
 * compares that register's four probe tests (8 of the probe's 64 bytes); a
 * state that passes is checked on every test by the warp.
 *
 * Bound: HBM latency and bandwidth, 45 bytes a state (a 32-byte sector of the
 * probe, task, rdl). A warp per state reading all live columns took 1.97 ms
 * for 5.3M states of 11 tests; this 0.06 ms. */
template <int TPC>
__global__ void __launch_bounds__(kThreads)
k_leaf_last(LevelDev P, TaskDev task, SolBuf S)
{
    const int lane = threadIdx.x & 31;
    const uint64_t n_round = (P.n + 31) & ~31ull;
    for (uint64_t q = (uint64_t)blockIdx.x * kThreads + threadIdx.x; q < n_round;
         q += (uint64_t)gridDim.x * kThreads) {
        uint32_t tid = 0, r = 0;
        bool pass = false;
        if (q < P.n) {
            tid = P.task[q];
            r = P.rdl[q];
            const uint2 v = *reinterpret_cast<const uint2 *>(P.probe + q * 32 + r * 4);
            const uint4 t = *reinterpret_cast<const uint4 *>(task.target + tid * 32);
            /* tests past the task's are zero in both */
            pass = task.active[tid] && r && v.x == (t.x | t.y << 16) && v.y == (t.z | t.w << 16);
        }
        uint32_t bal = __ballot_sync(0xFFFFFFFFu, pass);
        while (bal) {
            const int j = __ffs((int)bal) - 1;
            bal &= bal - 1;
            const unsigned long long qj = __shfl_sync(0xFFFFFFFFu, (unsigned long long)q, j);
            const uint32_t tj = __shfl_sync(0xFFFFFFFFu, tid, j);
            const uint32_t rj = __shfl_sync(0xFFFFFFFFu, r, j);
            const bool ok = lane >= task.T[tj] ||
                            P.regs[(qj * 8 + rj) * TPC + lane] == task.target[tj * 32 + lane];
            if (__all_sync(0xFFFFFFFFu, ok) && lane == 0) record(S, qj, 0, 0, rj, rj, 1);
        }
    }
}

/* Which of the ops of an operand-pair entry give t from (x, y): bit k < 9
   for the ALU op kPairOps[k], bit 9 for x + e (an ADDI, e its immediate
   sign-extended to 16 bits). Every op is evaluated, with no branch. */
__device__ __forceinline__ uint32_t pair_hits(uint32_t x, uint32_t y, uint32_t e, uint32_t t)
{
    const uint32_t s = y & 15u;
    uint32_t h = 0;
    h |= (uint32_t)(((x + y) & 0xFFFFu) == t);
    h |= (uint32_t)(((x - y) & 0xFFFFu) == t) << 1;
    h |= (uint32_t)(((x * y) & 0xFFFFu) == t) << 2;
    h |= (uint32_t)((x & y) == t) << 3;
    h |= (uint32_t)((x | y) == t) << 4;
    h |= (uint32_t)((x ^ y) == t) << 5;
    h |= (uint32_t)(((x << s) & 0xFFFFu) == t) << 6;
    h |= (uint32_t)((x >> s) == t) << 7;
    h |= (uint32_t)((uint32_t)(uint16_t)((int16_t)(uint16_t)x >> s) == t) << 8;
    h |= (uint32_t)(((x + e) & 0xFFFFu) == t) << 9;
    return h;
}

/* Scan the value classes of mask m against the warp's state, with operand
 * registers remapped: a register equal to rd2 reads spare column 9, else a
 * register equal to rd1 reads column 8 (rd = 8 means "none").
 *
 * need1 / need2 (0 = none): registers the last instruction must read. At a
 * depth K reached only after depth K-1 was searched without a solution,
 * every instruction of a solving program feeds a later one: an instruction
 * whose value nothing reads could be dropped, leaving a solving program of
 * K-1 instructions in the same candidate space. So the last instruction
 * reads the register the one before it wrote (need1), and need2 names an
 * earlier write nothing else read. Only classes that read need1 are
 * scanned, from the per-register class lists; the solutions are the same. */
template <int TPC, int FT>
__device__ __forceinline__ void scan_last(const WarpState<TPC> &ws, int T,
                                          uint32_t m, uint32_t rd1, uint32_t rd2, uint32_t tgt,
                                          uint32_t tgt0, uint32_t tgt1, uint32_t tgt2, int lane,
                                          const SolBuf &S, uint64_t q, uint32_t m1, uint32_t m2,
                                          uint32_t need1, uint32_t need2, unsigned long long &nev)
{
    if (need1) {
        /* the classes reading need1, one operand pair (or ADDI) per lane,
           every op of the pair evaluated on the first two tests at once */
        const uint32_t p0 = c_pr_off[m * 8 + need1], np = c_pr_off[m * 8 + need1 + 1] - p0;
        if (!need2 && lane == 0) nev += c_pr_ev[m * 8 + need1];
        for (uint32_t b0 = 0; b0 < np; b0 += 32) {
            const uint32_t i = b0 + lane;
            uint32_t hits = 0, ra = 0, rb = 0, e = 0;
            if (i < np) {
                const uint32_t d = c_pr[p0 + i];
                const uint32_t a = d & 7u, b = (d >> 3) & 7u;
                if (!need2 || a == need2 || b == need2) {
                    if (need2) nev += __popc((d >> 6) & 0x3FFu);
                    ra = a == rd2 ? 9u : a == rd1 ? 8u : a;
                    rb = b == rd2 ? 9u : b == rd1 ? 8u : b;
                    e = (uint32_t)(uint16_t)(int16_t)(int8_t)(uint8_t)(d >> 16);
                    hits = pair_hits(ws.R[ra][0], ws.R[rb][0], e, tgt0) & (d >> 6) & 0x3FFu;
                    if (FT >= 2 && T >= 2 && hits)
                        hits &= pair_hits(ws.R[ra][1], ws.R[rb][1], e, tgt1);
                    if (FT >= 3 && T >= 3 && hits)
                        hits &= pair_hits(ws.R[ra][2], ws.R[rb][2], e, tgt2);
                }
            }
            uint32_t bal = __ballot_sync(0xFFFFFFFFu, hits != 0);
            while (bal) {
                const int j = __ffs(bal) - 1;
                bal &= bal - 1;
                uint32_t hj = __shfl_sync(0xFFFFFFFFu, hits, j);
                const uint32_t aj = __shfl_sync(0xFFFFFFFFu, ra, j);
                const uint32_t bj = __shfl_sync(0xFFFFFFFFu, rb, j);
                const uint32_t ej = __shfl_sync(0xFFFFFFFFu, e, j);
                while (hj) {
                    const uint32_t k = (uint32_t)(__ffs(hj) - 1);
                    hj &= hj - 1;
                    bool ok = true;
                    if (lane < T) {
                        const uint32_t x = ws.R[aj][lane], y = ws.R[bj][lane];
                        ok = (k == 9 ? ((x + ej) & 0xFFFFu) : pca_alu(pair_op(k), x, y, 0)) == tgt;
                    }
                    if (__all_sync(0xFFFFFFFFu, ok) && lane == 0) {
                        const uint32_t cj = c_pr_cls[(uint64_t)(p0 + b0 + j) * 10 + k];
                        record_solution(S, q, m1, m2, cj, m);
                    }
                }
            }
        }
        return;
    }
    const uint32_t vbase = c_vc_off[m];
    const uint32_t *uops = c_vc_uop + vbase;
    const uint32_t nvc = c_vc_off[m + 1] - vbase;
    for (uint32_t b0 = 0; b0 < nvc; b0 += 32) {
        const uint32_t i = b0 + lane;
        uint32_t u = 0;
        bool pass = false;
        if (i < nvc) {
            /* the first FT tests per lane; survivors are checked on all tests below */
            u = uops[i];
            uint32_t ra = UOP_A(u), rb = UOP_B(u);
            const bool reads2 = !need2 || ra == need2 || rb == need2;
            ra = ra == rd2 ? 9u : ra == rd1 ? 8u : ra;
            rb = rb == rd2 ? 9u : rb == rd1 ? 8u : rb;
            const uint32_t op = UOP_OP(u), imm = UOP_IMM(u);
            nev += reads2 ? 1u : 0u;
            pass = reads2 && pca_alu(op, ws.R[ra][0], ws.R[rb][0], imm) == tgt0 &&
                   (FT < 2 || T < 2 || pca_alu(op, ws.R[ra][1], ws.R[rb][1], imm) == tgt1) &&
                   (FT < 3 || T < 3 || pca_alu(op, ws.R[ra][2], ws.R[rb][2], imm) == tgt2);
        }
        uint32_t bal = __ballot_sync(0xFFFFFFFFu, pass);
        while (bal) {
            const int j = __ffs(bal) - 1;
            bal &= bal - 1;
            const uint32_t uj = __shfl_sync(0xFFFFFFFFu, u, j);
            uint32_t ra = UOP_A(uj), rb = UOP_B(uj);
            ra = ra == rd2 ? 9u : ra == rd1 ? 8u : ra;
            rb = rb == rd2 ? 9u : rb == rd1 ? 8u : rb;
            bool ok = true;
            if (lane < T) ok = pca_alu(UOP_OP(uj), ws.R[ra][lane], ws.R[rb][lane], UOP_IMM(uj)) == tgt;
            if (__all_sync(0xFFFFFFFFu, ok) && lane == 0) record_solution(S, q, m1, m2, b0 + j, m);
        }
    }
}

/* The suffix kernels' view of a prefix: only its live columns (no operand
   of a candidate reads anything else; column 0 is zeroed once per warp)
   and no flags (no branchless op reads them). */
template <int TPC>
__device__ __forceinline__ void load_live_cols(WarpState<TPC> &ws, const uint16_t *regs,
                                               uint64_t q, uint32_t live, int lane)
{
    if (lane < TPC) {
        const uint16_t *src = regs + q * 8 * TPC + lane;
#pragma unroll
        for (int r = 1; r < 8; r++)
            if ((live >> r) & 1u) ws.R[r][lane] = src[r * TPC];
    }
}

/* A contiguous range of prefixes, optionally through a permutation: the
 * suffix kernel visits prefixes order[begin .. begin + count) (or begin ..
 * begin + count when order is null). */
/* Counts entries of order[0..n) that are >= n or repeat an earlier value
 * (seen: zeroed bitmap of n bits). Zero means order is a permutation. */
__global__ void k_check_perm(const uint32_t *order, uint64_t n, uint32_t *seen,
                             unsigned long long *bad)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = order[i];
        if (v >= n) {
            atomicAdd(bad, 1ull);
            continue;
        }
        const uint32_t bit = 1u << (v & 31);
        if (atomicOr(&seen[v >> 5], bit) & bit) atomicAdd(bad, 1ull);
    }
}

struct PrefixRange {
    const uint32_t *order;
    uint64_t begin, count;
};

/* Suffix enumeration of depth SD (1..3) from the prefixes of level P in
 * range R whose task is active. Work item = (prefix, chunk of first-suffix
 * candidates); for SD = 1 the chunk is the whole prefix. Five CTAs per SM
 * (48 registers) measured fastest: at SD = 1 four CTAs at 64 registers hide
 * less latency and six spill the prefetched columns; at SD = 2 five CTAs
 * instead of the four that 56 registers allow cut a two-input depth-4
 * stage from 39 to 30 ms. */
template <int TPC, int SD, int FT>
__global__ void __launch_bounds__(kThreads, 5)
k_suffix(LevelDev P, TaskDev task, SolBuf S, uint32_t chunks_per_prefix, uint32_t chunk,
         PrefixRange R)
{
    __shared__ WarpState<TPC> sws[kWarpsPerBlock];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    WarpState<TPC> &ws = sws[wib];
    const uint64_t nw = (uint64_t)gridDim.x * kWarpsPerBlock;
    const uint64_t items = R.count * chunks_per_prefix;
    uint64_t loaded = ~0ull;
    uint32_t cur_task = ~0u, tgt = 0, tgt0 = 0, tgt1 = 0, tgt2 = 0;
    int T = 0;
    unsigned long long nev = 0;
    if (lane < TPC) ws.R[0][lane] = 0;
    bool cur_active = false;
    if constexpr (SD == 1) {
        /* one prefix per item, software-pipelined: the next prefix's
           links and columns are loaded while this one's classes are scanned
           (the scan is short, and waiting on those loads bounded the loop) */
        uint64_t nq = ~0ull;
        uint32_t ntid = 0, nlive = 0, nw0 = 0, ncol[7];
        auto fetch = [&](uint64_t i) {
            nq = ~0ull;
            if (i >= items) return;
            const uint64_t q = R.order ? (uint64_t)R.order[R.begin + i] : R.begin + i;
            if (q >= P.n) return;  /* orders are checked on the host; never index outside */
            nq = q;
            ntid = P.task[q];
            nlive = P.live[q];
            nw0 = P.rdl[q];
            const uint16_t *src = P.regs + q * 8 * TPC + (lane < TPC ? lane : 0);
#pragma unroll
            for (int r = 1; r < 8; r++) ncol[r - 1] = src[r * TPC];
        };
        uint64_t it = (uint64_t)blockIdx.x * kWarpsPerBlock + wib;
        fetch(it);
        for (; it < items; it += nw) {
            const uint64_t q = nq;
            const uint32_t tid = ntid, live = nlive, w0 = nw0;
            if (q != ~0ull) {
                __syncwarp();
                if (lane < TPC) {
#pragma unroll
                    for (int r = 1; r < 8; r++) ws.R[r][lane] = ncol[r - 1];
                }
                __syncwarp();
            }
            fetch(it + nw);
            if (q == ~0ull) continue;
            if (tid != cur_task) {
                cur_task = tid;
                cur_active = task.active[tid] != 0;
                T = task.T[tid];
                tgt = lane < T ? task.target[tid * 32 + lane] : 0u;
                tgt0 = task.target[tid * 32];
                tgt1 = task.target[tid * 32 + 1];
                if (FT >= 3) tgt2 = task.target[tid * 32 + 2];
            }
            if (!cur_active) continue;
            /* w0: the prefix's last write (0 at a root); some later
               instruction must read it (the rule scan_last states) */
            scan_last<TPC, FT>(ws, T, (live >> 1) & 127u, 8, 8, tgt, tgt0, tgt1, tgt2, lane, S, q, 0, 0, w0,
                           0, nev);
        }
        /* no flush: k_count_evals counts this depth's evaluations (nev is
           dead here and costs no register) */
        return;
    }
    for (uint64_t it = (uint64_t)blockIdx.x * kWarpsPerBlock + wib; it < items; it += nw) {
        const uint64_t qi = it / chunks_per_prefix;
        const uint32_t ck = (uint32_t)(it - qi * chunks_per_prefix);
        const uint64_t q = R.order ? (uint64_t)R.order[R.begin + qi] : R.begin + qi;
        if (q >= P.n) continue;  /* orders are checked on the host; never index outside */
        const uint32_t tid = P.task[q];
        if (tid != cur_task) {
            cur_task = tid;
            cur_active = task.active[tid] != 0;
            T = task.T[tid];
            tgt = lane < T ? task.target[tid * 32 + lane] : 0u;
            tgt0 = task.target[tid * 32];
            tgt1 = task.target[tid * 32 + 1];
            if (FT >= 3) tgt2 = task.target[tid * 32 + 2];
        }
        if (!cur_active) continue;
        const uint32_t live = P.live[q];
        if (q != loaded) {
            __syncwarp();
            load_live_cols<TPC>(ws, P.regs, q, live, lane);
            loaded = q;
            __syncwarp();
        }
        const uint32_t m0 = (live >> 1) & 127u;
        /* the prefix's last write (0 at a root): some later instruction
           must read it (the rule scan_last states) */
        const uint32_t w0 = P.rdl[q];
        const uint32_t cb0 = c_cand_off[m0], nc0 = c_cand_off[m0 + 1] - cb0;
        const uint32_t lo = ck * chunk, hi = min(nc0, lo + chunk);
        for (uint32_t i1 = lo; i1 < hi; i1++) {
            const uint32_t u1 = c_cand_uop[cb0 + i1];
            /* a middle writing the same value and flags as an earlier
               sibling leads to the states that sibling leads to: under OEP
               its subtree is the pruned duplicate (never the DFS-first) */
            if (task.dedup_mid && (u1 >> 31)) continue;
            const uint32_t rd1 = UOP_RD(u1);
            /* w0 still unread after u1: overwritten (dead, skip) or owed by
               a later instruction */
            const uint32_t owe0 = w0 && !uop_reads(u1, w0) ? w0 : 0u;
            if (owe0 && rd1 == owe0) continue;
            __syncwarp();
            if (lane < TPC)
                ws.R[8][lane] = lane < T ? pca_alu(UOP_OP(u1), ws.R[UOP_A(u1)][lane],
                                                   ws.R[UOP_B(u1)][lane], UOP_IMM(u1))
                                         : 0u;
            __syncwarp();
            const uint32_t m1 = (m0 | (1u << (rd1 - 1))) & 127u;
            if (SD == 2) {
                scan_last<TPC, FT>(ws, T, m1, rd1, 8, tgt, tgt0, tgt1, tgt2, lane, S, q, i1, 0, rd1, owe0,
                               nev);
                continue;
            }
            const uint32_t cb1 = c_cand_off[m1], nc1 = c_cand_off[m1 + 1] - cb1;
            for (uint32_t i2 = 0; i2 < nc1; i2++) {
                const uint32_t u2 = c_cand_uop[cb1 + i2];
                if (task.dedup_mid && (u2 >> 31)) continue;
                const uint32_t rd2 = UOP_RD(u2);
                /* writes still owed a read after u2 (u1's and maybe w0's);
                   one overwritten unread is dead, and the last instruction
                   reads rd2 and at most one more register */
                const uint32_t owe1 = uop_reads(u2, rd1) ? 0u : rd1;
                const uint32_t owe0b = owe0 && !uop_reads(u2, owe0) ? owe0 : 0u;
                if ((owe1 && rd2 == owe1) || (owe0b && rd2 == owe0b)) continue;
                if (owe1 && owe0b) continue;   /* three registers to read */
                const uint32_t need2 = owe1 ? owe1 : owe0b;
                uint32_t ra = UOP_A(u2), rb = UOP_B(u2);
                ra = ra == rd1 ? 8u : ra;
                rb = rb == rd1 ? 8u : rb;
                __syncwarp();
                if (lane < TPC)
                    ws.R[9][lane] = lane < T ? pca_alu(UOP_OP(u2), ws.R[ra][lane],
                                                       ws.R[rb][lane], UOP_IMM(u2))
                                             : 0u;
                __syncwarp();
                const uint32_t m2 = (m1 | (1u << (rd2 - 1))) & 127u;
                scan_last<TPC, FT>(ws, T, m2, rd2 == rd1 ? 8u : rd1, rd2, tgt, tgt0, tgt1, tgt2, lane, S,
                               q, i1, i2, rd2, need2, nev);
            }
        }
    }
    flush_evals(S, nev, lane);
}

}  // namespace pcagb

#include "suffix_forms.cuh"

namespace pcagb {

/* Value-class evaluations k_suffix<TPC, 1> runs over range R: a prefix of
   mask m whose last write is w0 scans the pair list of (m, w0), a root
   every class of its mask (c_ev_sd1, in global memory: the lanes read
   different entries). Added to S.evals, one atomic per warp. */
__global__ void k_count_evals(LevelDev P, TaskDev task, PrefixRange R, SolBuf S)
{
    const int lane = threadIdx.x & 31;
    unsigned long long nev = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t n_round = (R.count + 31) & ~31ull;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_round; i += stride) {
        if (i >= R.count) continue;
        const uint64_t q = R.order ? (uint64_t)R.order[R.begin + i] : R.begin + i;
        if (q >= P.n || !task.active[P.task[q]]) continue;
        const uint32_t m = (P.live[q] >> 1) & 127u, w0 = P.rdl[q];
        nev += __ldg(c_ev_sd1 + m * 8 + w0);
    }
    flush_evals(S, nev, lane);
}

/* ---- recording: the reference's keys and records of level states --------- */

/* Engine column of each original test (the engine reorders tests). */
struct TestPos {
    uint8_t pos[MAX_TESTS];
};

/* FNV-1a-64 over the state's bytes in the reference's order (per original
 * test: r0..r7 low byte then high byte, then the flags): the oep hash; the
 * key adds live and depth (src/search_state.c:191-219). One thread per
 * state. */
template <int TPC>
__global__ void k_record_keys(LevelDev L, TestPos tp, int T, int depth, uint64_t *key,
                              uint64_t *oep)
{
    const uint64_t prime = 0x00000100000001B3ull;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < L.n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t h = 0xCBF29CE484222325ull;
        for (int u = 0; u < T; u++) {
            const int c = tp.pos[u];
#pragma unroll
            for (int r = 0; r < 8; r++) {
                const uint32_t v = L.regs[(i * 8 + r) * TPC + c];
                h = (h ^ (v & 0xFFu)) * prime;
                h = (h ^ (v >> 8)) * prime;
            }
            h = (h ^ L.flags[i * TPC + c]) * prime;
        }
        oep[i] = h;
        h = (h ^ L.live[i]) * prime;
        h = (h ^ (uint32_t)depth) * prime;
        key[i] = h;
    }
}

/* What the recording pass writes for one state (src/search_state.c:243-268). */
struct RecordMeta {
    uint32_t index;          /* state in its level */
    uint16_t parent_action;  /* 0xFFFF for the root */
    uint8_t  positive;
    int8_t   remaining;
};

/* One warp per record, lane = original test; `out` is zeroed beforehand. */
template <int TPC>
__global__ void k_record_states(LevelDev L, TestPos tp, int T, int depth, uint32_t task_id,
                                int target_depth, const RecordMeta *meta, uint64_t count,
                                const uint64_t *key, const uint64_t *oep,
                                dataset_state_record_t *out)
{
    const int lane = threadIdx.x & 31;
    const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < count; w += nw) {
        const RecordMeta m = meta[w];
        const uint64_t i = m.index;
        dataset_state_record_t &o = out[w];
        if (lane == 0) {
            o.state_hash = key[i];
            o.oep_hash = oep[i];
            o.task_id = task_id;
            o.parent_action = m.parent_action;
            o.depth = (uint8_t)depth;
            o.budget_left = (uint8_t)(target_depth - depth);
            o.live = L.live[i];
            o.can_finish_optimally = m.positive;
            o.remaining_steps = m.remaining;
        }
        if (lane < T) {
            const int c = tp.pos[lane];
#pragma unroll
            for (int r = 0; r < 8; r++) o.regs[lane][r] = L.regs[(i * 8 + r) * TPC + c];
            o.flags[lane] = L.flags[i * TPC + c];
        }
    }
}

}  // namespace pcagb
