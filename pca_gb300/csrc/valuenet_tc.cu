/*
 * valuenet_tc.cu -- the value network's per-test encoder on the fifth-
 * generation tensor cores (tcgen05 + TMEM + TMA), fused from the level's
 * states to the pooled state vector.
 *
 * One persistent pair of CTAs (a cluster of two on neighbouring SMs) walks
 * tiles of 256 feature rows: 8 states x 32 test rows, 4 states a CTA. Both
 * layers are tcgen05.mma.cta_group::2 products (M = 256, N = 256, K = 16,
 * BF16 in, FP32 accumulate), so each SM keeps half of the weights: its 128
 * units of W1 and of W2 (112 KB) are loaded once by TMA and stay in shared
 * memory for every tile. Per tile, in each CTA:
 *   features  the 176 bit features of each of its (state, test) rows (the
 *             columns of k_features in valuenet.cu), expanded to BF16 in
 *             registers straight into the swizzled K-major operand A1;
 *   layer E1  A1 x W1^T: TMEM lanes = the CTA's 128 rows, columns 0..255 =
 *             the units;
 *   epi 1     tcgen05.ld, + bias, ReLU and BF16 rounding in one packed
 *             convert, held in registers until the previous tile's E2 has
 *             read A2, then stored there (swizzled, K-major);
 *   layer E2  W2 x A2^T, the operands exchanged: TMEM lanes = the CTA's 128
 *             units, columns 256..511 = the pair's 256 rows;
 *   epi 2     each lane owns a unit: + bias, ReLU, BF16, the sum (fp32,
 *             tests in order) and the maximum over a state's T columns, all
 *             in registers, and writes P[528] = mean(256) | max(256) | live
 *             bits(8) | depth | zeros -- the values of k_pool on the same
 *             H2. H2 is written nowhere.
 * The activations X, H1 and H2 never reach HBM: per state the kernel reads
 * the level record (17 x T bytes) and writes 1,056 bytes.
 *
 * Roles: warp 0's first thread loads the weights; warp 1 owns TMEM and, in
 * the first CTA, one of its threads issues every MMA; eight front warps
 * write the features and E1's epilogue, eight back warps E2's (two warps
 * each per TMEM lane quarter). E1 is issued as two halves of 128 units, so
 * that the front starts on the first while the second runs. The MMAs run in
 * the order E1(i + 1), E2(i): the front's work on tile i + 1 and the
 * features of tile i + 2 run while E2(i) does, the back's on tile i while
 * E1(i + 2) does.
 *
 * What bounds it: 27 MMAs of 128 cycles a tile, 3,456, and the hand-overs
 * between the roles: 5,300 cycles a tile, tensor pipe 65% busy. In the
 * one-CTA form (weights streamed, H2 pooled through shared memory by the
 * same 16 warps) the operands, 224 KB of weight slabs a tile and H2's way
 * were 800 KB of shared-memory traffic a tile of 128 rows and each warp
 * waited for its own record loads, 10,900 cycles. Measured on the way
 * (131,072 states of 16 to 32 tests): the pair alone 1.21 -> 0.85 ms; front
 * and back apart, accumulators fetched ahead and nothing computed from a
 * record when it is loaded 0.67; the quotient below and E1 in halves 0.63;
 * descriptors not kept 0.60. 4,096 states: 47 -> 31 us.
 *
 * Synchronisation is by mbarriers (and one cluster barrier at each end);
 * every wait is bounded by the global timer (kWaitNs). A wait that runs out
 * sets the CTA's abort flag and the status word, every role of the CTA
 * leaves its loop, and the other CTA's waits run out in turn; the MMA thread
 * waits for its own MMAs, and TMEM is freed once both CTAs are done.
 */
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "../../include/pca_gb300.h"
#include "per_device.h"

namespace {

constexpr int kRows = 128;            /* feature rows per CTA and tile */
constexpr int kStatesPerTile = 8;     /* of a pair */
constexpr int kUnits = 256;           /* units of both encoder layers */
constexpr int kHalfUnits = kUnits / 2; /* of one CTA's weights */
constexpr int kFeat = 176;            /* feature columns (164 used) */
constexpr int kKB1 = 3, kKB2 = 4;     /* 64-column K blocks of E1 (176 of 192) and E2 */
constexpr int kFrontWarps = 8, kBackWarps = 8;
constexpr int kThreads = 64 + 32 * (kFrontWarps + kBackWarps); /* warp 0 TMA, 1 MMA + TMEM */
constexpr int kBlock = kRows * 128;   /* 16 KB: 128 rows x 64 bf16 of any operand */
constexpr int kOffA1 = 0;                             /* 48 KB */
constexpr int kOffA2 = kOffA1 + kKB1 * kBlock;        /* 64 KB */
constexpr int kOffW1 = kOffA2 + kKB2 * kBlock;        /* 48 KB */
constexpr int kOffW2 = kOffW1 + kKB1 * kBlock;        /* 64 KB */
constexpr int kOffBias = kOffW2 + kKB2 * kBlock;      /* b1: 256 fp32 */
constexpr int kOffBar = kOffBias + kUnits * 4;
constexpr int kSmemBytes = kOffBar + 256 + 1024;      /* + alignment slack */
constexpr int kPoolCols = 528;
constexpr unsigned long long kWaitNs = 1000000000ull; /* 1 s per wait */
static_assert(kRows == kHalfUnits, "A and B blocks are the same size");
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

/* barrier slots (8 bytes each). Counted in the pair's first CTA (an arrival
   per front or back warp of both): A1 and A2 written, the halves of D1 and
   D2 drained. In each CTA: weights landed, E1's halves done (the second: A1
   read), E2's four K blocks done (that block of A2 read; the last one: D2
   complete), all MMAs done. */
constexpr int kBarA1 = 0, kBarA2 = 1, kBarFree1 = 2, kBarFree2 = 4, kBarW = 5, kBarD1 = 6,
              kBarE2 = 8, kBarDrain = kBarE2 + kKB2, kBarCount = kBarDrain + 1;
constexpr int kOffTmemSlot = kBarCount * 8;
constexpr int kOffAbort = kOffTmemSlot + 4;
static_assert(kOffAbort + 4 <= 256, "barrier area");

/* Instruction descriptor of tcgen05.mma kind::f16: D f32 (bits 4-5 = 1),
   A and B bf16 (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bits 17-22,
   M >> 4 at bits 24-28. Of the pair: M = 256, N = 128 (E1, a half of the
   units) or 256 (E2). */
constexpr uint32_t kIdescM256 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 4) << 24);
constexpr uint32_t kIdescE1 = kIdescM256 | ((uint32_t)(kHalfUnits >> 3) << 17);
constexpr uint32_t kIdescE2 = kIdescM256 | ((uint32_t)(2 * kRows >> 3) << 17);

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

/* arrive on the barrier at this offset of the cluster's first CTA */
__device__ __forceinline__ void mbar_arrive_first(uint32_t bar)
{
    asm volatile(
        "{\n\t.reg .b32 ra;\n\t"
        "mapa.shared::cluster.u32 ra, %0, 0;\n\t"
        "mbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}" ::"r"(bar)
        : "memory");
}

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

/* Wait for the phase of `parity` to complete, at most kWaitNs; on time-out
   (or an abort raised elsewhere) set the abort flag and return false. */
__device__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status,
                          int code)
{
    if (mbar_test(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (uint32_t i = 0;; i++) {
        if (mbar_test(bar, parity)) return true;
        if ((i & 15) == 15) {
            if (*abort_flag) return false;
            if (global_ns() - t0 > kWaitNs) {
                *abort_flag = 1;
                atomicExch(status, code);
                return false;
            }
        }
    }
}

__device__ __forceinline__ void fence_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar,
                                            int x, int y)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y)
        : "memory");
}

/* Shared-memory matrix descriptor: K-major operand in 128-byte swizzle
   atoms (8 rows x 128 B), 8-row groups 1024 B apart; the address in the low
   word. */
constexpr uint64_t kSw128Desc = (uint64_t)1 << 16 |            /* leading byte offset: unused */
                                (uint64_t)(1024 >> 4) << 32 |  /* stride byte offset */
                                (uint64_t)1 << 46 |            /* descriptor version */
                                (uint64_t)2 << 61;             /* 128-byte swizzle */

__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr)
{
    return kSw128Desc | (uint64_t)((saddr & 0x3FFFFu) >> 4);
}

/* Shared-memory matrix descriptor: MN-major operand in 128-byte swizzle
   atoms (8 K-rows x 128 B = 64 elements along M or N), 8-row groups 1024 B
   apart along K, 64-element groups along M or N 8 KB apart (one 64 x 64
   TMA box each). */
__device__ __forceinline__ uint64_t sw128_mn_desc(uint32_t saddr)
{
    uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(8192 >> 4) << 16;  /* leading byte offset: next 64 along M/N */
    d |= (uint64_t)(1024 >> 4) << 32;  /* stride byte offset: next 8 along K */
    d |= (uint64_t)1 << 46;            /* descriptor version */
    d |= (uint64_t)2 << 61;            /* 128-byte swizzle */
    return d;
}

/* one product of the pair: A and B at these offsets of both CTAs, given as
   the low words of their descriptors */
__device__ __forceinline__ void mma_pair(uint32_t dtmem, uint32_t a, uint32_t b, uint32_t idesc,
                                         uint32_t acc)
{
    constexpr uint32_t high = (uint32_t)(kSw128Desc >> 32);
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(dtmem),
        "r"(a), "r"(b), "r"(idesc), "r"(acc), "r"(high)
        : "memory");
}

/* arrive on the barrier at this offset of both CTAs of the pair once the
   thread's products so far are done */
__device__ __forceinline__ void mma_commit_pair(uint32_t bar)
{
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
        "[%0], %1;" ::"r"(bar), "h"((uint16_t)3)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
        : "memory");
}

/* 32 columns of this warp's lanes into registers; r is not to be read before
   tmem_wait(r) */
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait(uint32_t (&r)[32])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]),
                   "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                   "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
                   "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32])
{
    tmem_ld32_async(taddr, r);
    tmem_wait(r);
}

/* Byte offset of 16-byte chunk c (0..7) of row r in a 128-byte-swizzled
   block (the layout TMA's 128B swizzle writes and the descriptor reads). */
__device__ __forceinline__ uint32_t sw128_off(int r, int c)
{
    return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4));
}

/* 8 bits of a 16-bit word w (the low or the high byte) as 8 bf16 values 0.0 /
   1.0, the byte's bit 0 first. y has the byte's bit 2j at 2j and bit 2j + 1
   at 16 + 2j; the two, times 0x3F80 >> 2j, are the halves of output word j. */
__device__ __forceinline__ uint4 byte_to_bf16x8(uint32_t w, int high)
{
    const uint32_t y = high ? (w >> 8) | (w << 7) : w | (w << 15);
    return make_uint4((y & 0x00010001u) * 0x3F80u, (y & 0x00040004u) * (0x3F80u >> 2),
                      (y & 0x00100010u) * (0x3F80u >> 4), (y & 0x00400040u) * (0x3F80u >> 6));
}

/* v / T rounded to nearest, v >= 0 and 1 <= T <= 32 (T = 0: v is 0), with
   r = 1 / T rounded to nearest: Markstein's correction of a quotient
   (Computation of elementary functions on the IBM RISC System/6000
   processor, 1990). Away from the ends of the range its steps scale with v,
   and over all 2^23 significands and each T it gives the division's value;
   at the ends it is the division. A division for each of the four sums of a
   lane takes 1,400 cycles of a tile beside the other warps, this a tenth. */
__device__ __forceinline__ float quotient(float v, int T, float r)
{
    if (v > 0.f && !(v > 1e-30f && v < 1e38f)) return v / (float)T;
    const float q = v * r;
    return __fmaf_rn(__fmaf_rn(-(float)T, q, v), r, q);
}

/* s + the low half + the high half of x, in this order */
__device__ __forceinline__ float add_bf16x2(float s, uint32_t x)
{
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\t"
        "add.rn.f32.bf16 %0, l, %0;\n\tadd.rn.f32.bf16 %0, h, %0;\n\t}"
        : "+f"(s)
        : "r"(x));
    return s;
}

/* (a.x + b.x, a.y + b.y), each rounded as a single addition */
__device__ __forceinline__ float2 add_f32x2(uint32_t ax, uint32_t ay, float bx, float by)
{
    float2 d;
    asm("{\n\t.reg .b64 a, b, c;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "add.rn.f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "r"(ax), "r"(ay), "f"(bx), "f"(by));
    return d;
}

/* relu(lo), relu(hi) rounded to bf16, lo in the low half. */
__device__ __forceinline__ uint32_t relu_bf16x2(float lo, float hi)
{
    uint32_t d;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b)
{
    uint32_t d;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
k_encode_pool_tc(const __grid_constant__ CUtensorMap map_w1, const __grid_constant__ CUtensorMap map_w2,
                 const float *__restrict__ b1, const float *__restrict__ b2,
                 const uint16_t *__restrict__ regs, const uint8_t *__restrict__ flags,
                 const uint8_t *__restrict__ live, const uint16_t *__restrict__ task,
                 const uint8_t *__restrict__ depth, int TP, int n,
                 const uint16_t *__restrict__ task_io, const int32_t *__restrict__ task_T,
                 __nv_bfloat16 *__restrict__ P, int *status)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sA1 = smem_u32(smem + kOffA1), sA2 = smem_u32(smem + kOffA2);
    const uint32_t sW1 = smem_u32(smem + kOffW1), sW2 = smem_u32(smem + kOffW2);
    const uint32_t sBar = smem_u32(smem + kOffBar);
    uint32_t *tmem_slot = (uint32_t *)(smem + kOffBar + kOffTmemSlot);
    volatile int *abort_flag = (volatile int *)(smem + kOffBar + kOffAbort);
    float *sb1 = (float *)(smem + kOffBias);
    auto bar = [&](int i) { return sBar + 8u * (uint32_t)i; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1;                     /* in the pair */
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int ntiles = (n + kStatesPerTile - 1) / kStatesPerTile;
    const int mine = pair < ntiles ? (ntiles - 1 - pair) / pairs + 1 : 0;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kBarCount; i++)
            mbar_init(bar(i), i < kBarFree2 ? 2 * kFrontWarps : i == kBarFree2 ? 2 * kBackWarps : 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
        mbar_expect_tx(bar(kBarW), (kKB1 + kKB2) * kBlock);
        for (int k = 0; k < kKB1; k++)
            for (int u = 0; u < 2; u++)      /* its quarter of each half of the units */
                tma_load_2d(sW1 + k * kBlock + u * (kBlock / 2), &map_w1, bar(kBarW), 64 * k,
                            kHalfUnits * u + kHalfUnits / 2 * rank);
        for (int k = 0; k < kKB2; k++)
            tma_load_2d(sW2 + k * kBlock, &map_w2, bar(kBarW), 64 * k, kHalfUnits * rank);
    }
    for (int i = threadIdx.x; i < kUnits; i += kThreads) sb1[i] = b1[i];
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                         smem_u32(tmem_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *tmem_slot;
    /* both CTAs' barriers are set up, their TMEM is theirs, their weights
       have landed */
    mbar_wait(bar(kBarW), 0, abort_flag, status, 1);
    __syncwarp();
    cluster_sync();

    if (warp == 1) {
        /* ---- MMA issuer (first CTA) ---- */
        if (lane == 0 && rank == 0) {
            auto wait = [&](int which, int tile, int code) {
                return mbar_wait(bar(which), tile & 1, abort_flag, status, code);
            };
            /* Unrolled: a product takes this thread 100 cycles to issue, in
               a loop 190, longer than the tensor core needs. The descriptors'
               low words are hidden from the compiler at each use: it would
               otherwise keep all 76 of them, and load many back from local
               memory before their product (633 us; so 601). */
            const uint32_t a1 = (uint32_t)sw128_desc(sA1), w1 = (uint32_t)sw128_desc(sW1);
            const uint32_t a2 = (uint32_t)sw128_desc(sA2), w2 = (uint32_t)sw128_desc(sW2);
            auto hidden = [](uint32_t v) {
                asm volatile("" : "+r"(v));
                return v;
            };
            /* K step k of 16: 32 bytes along the rows of a 64-column block */
            auto step = [](int k) { return (uint32_t)((k >> 2) * (kBlock >> 4) + (k & 3) * 2); };
            auto e1 = [&](int i) {
                if (!wait(kBarA1, i, 2)) return false;
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    if (i && !wait(kBarFree1 + u, i - 1, 3)) return false;
                    tc_after();
                    const uint32_t a = hidden(a1), w = hidden(w1 + u * (kBlock >> 5));
#pragma unroll
                    for (int k = 0; k < kFeat / 16; k++)
                        mma_pair(tmem + kHalfUnits * u, a + step(k), w + step(k), kIdescE1, k != 0);
                    mma_commit_pair(bar(kBarD1 + u));
                }
                return true;
            };
            auto e2 = [&](int i) {
                if (!wait(kBarA2, i, 4)) return false;
                if (i && !wait(kBarFree2, i - 1, 5)) return false;
                tc_after();
                const uint32_t a = hidden(a2), w = hidden(w2);
#pragma unroll
                for (int k = 0; k < 4 * kKB2; k++) {
                    mma_pair(tmem + kUnits, w + step(k), a + step(k), kIdescE2, k != 0);
                    if ((k & 3) == 3) mma_commit_pair(bar(kBarE2 + (k >> 2)));
                }
                return true;
            };
            bool ok = mine > 0 && e1(0);
            for (int i = 0; i < mine && ok; i++) {
                if (i + 1 < mine) ok = e1(i + 1);
                ok = ok && e2(i);
            }
            /* every MMA this thread issued has finished before TMEM is freed */
            mma_commit_pair(bar(kBarDrain));
            const unsigned long long t0 = global_ns();
            while (!mbar_test(bar(kBarDrain), 0) && global_ns() - t0 < kWaitNs) {
            }
        }
    } else if (warp >= 2 && warp < 2 + kFrontWarps) {
        /* ---- front warps: features, and E1's epilogue into A2 ---- */
        const int q = warp & 3;              /* TMEM lane quarter = the CTA's state */
        const int h = (warp - 2) >> 2;       /* its K blocks of A2: h and h + 2 */
        const int r = q * 32 + lane;         /* row of A1 and A2 = TMEM lane */
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;

        /* A state's level record, loaded one tile ahead of its features:
           the 16-bit words of this warp's half of the feature row (h = 0:
           in0 in1 target r1 r2 r3; 1: r4 r5 r6 r7 flags) for test `lane`,
           the task's tests and (h = 0, lanes 0..15) the pooled row's tail.
           The task id is loaded a tile earlier still and nothing is computed
           from what was loaded until its tile, so nothing in the loop waits
           for a load. */
        struct Rec {
            int s, T;
            uint32_t w[6];
            uint32_t g;  /* lane < 8: live mask, 8: depth, else 0 */
        };
        auto own = [&](int i) {
            return i < mine ? (pair + i * pairs) * kStatesPerTile + 4 * rank + q : n;
        };
        auto task_of = [&](int s) -> int { return s < n ? (int)task[s] : -1; };
        auto load_rec = [&](int i, int tid, Rec &rc) {
            rc.s = own(i);
            rc.T = 0;
            rc.g = 0;
#pragma unroll
            for (int k = 0; k < 6; k++) rc.w[k] = 0;
            if (tid < 0) return;
            rc.T = task_T[tid];
            if (h == 0 && lane < 9) rc.g = (lane < 8 ? live : depth)[rc.s];
            if (lane >= TP) return;
            const uint16_t *rg = regs + (size_t)rc.s * 8 * TP + lane;
            if (h == 0) {
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    rc.w[k] = task_io[((size_t)tid * 3 + k) * 32 + lane];
                    rc.w[3 + k] = rg[(1 + k) * TP];
                }
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) rc.w[k] = rg[(4 + k) * TP];
                rc.w[4] = flags[(size_t)rc.s * TP + lane];
            }
        };
        /* bit features of (state, test lane), this half's chunks of the
           row's 22 16-byte chunks, into A1 (rows past the task's tests are
           zero), and the pooled row's tail */
        auto features = [&](const Rec &rc) {
            const bool valid = lane < rc.T;
#pragma unroll
            for (int k = 0; k < 12; k++) {
                const int c = 12 * h + k;
                if (c >= kFeat / 8) break;
                *(uint4 *)(smem + kOffA1 + (c >> 3) * kBlock + sw128_off(r, c & 7)) =
                    byte_to_bf16x8(!valid ? 0u : c >= 20 ? rc.w[k >> 1] & 0xFu : rc.w[k >> 1],
                                   k & 1);
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive_first(bar(kBarA1));
            if (h == 0 && lane < 16 && rc.s < n)
                P[(size_t)rc.s * kPoolCols + 2 * kUnits + lane] =
                    __float2bfloat16((float)(lane < 8 ? (rc.g >> lane) & 1u : rc.g));
        };

        /* a K block (64 units) of E1: + bias, ReLU, bf16, into registers */
        auto drain = [&](int kb, uint32_t (&w)[32]) {
#pragma unroll
            for (int g = 0; g < 2; g++) {
                uint32_t acc[32];
                tmem_ld32(tmem + lane_base + (uint32_t)(64 * kb + 32 * g), acc);
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const float4 b = *(const float4 *)(sb1 + 64 * kb + 32 * g + 4 * c);
                    const float2 u = add_f32x2(acc[4 * c], acc[4 * c + 1], b.x, b.y);
                    const float2 v = add_f32x2(acc[4 * c + 2], acc[4 * c + 3], b.z, b.w);
                    w[16 * g + 2 * c] = relu_bf16x2(u.x, u.y);
                    w[16 * g + 2 * c + 1] = relu_bf16x2(v.x, v.y);
                }
            }
        };

        Rec rec;
        load_rec(0, task_of(own(0)), rec);
        int tid_next = task_of(own(1));
        if (mine) features(rec);
        load_rec(1, tid_next, rec);
        tid_next = task_of(own(2));
        for (int i = 0; i < mine; i++) {
            bool ok = true;
#pragma unroll 1
            for (int u = 0; u < 2; u++) {
                const int kb = 2 * u + h;
                uint32_t w[32];
                ok = mbar_wait(bar(kBarD1 + u), i & 1, abort_flag, status, 6);
                if (!__all_sync(0xffffffffu, ok)) break;
                tc_after();
                drain(kb, w);
                tc_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_first(bar(kBarFree1 + u));
                if (u == 0) {
                    /* E1 has read A1 once its second half is done: the next
                       tile's features */
                    ok = mbar_wait(bar(kBarD1 + 1), i & 1, abort_flag, status, 6);
                    if (!__all_sync(0xffffffffu, ok)) break;
                    if (i + 1 < mine) features(rec);
                }
                /* into A2 once the previous tile's E2 has read the block */
                if (i) {
                    ok = mbar_wait(bar(kBarE2 + kb), (i - 1) & 1, abort_flag, status, 7);
                    if (!__all_sync(0xffffffffu, ok)) break;
                }
#pragma unroll
                for (int c = 0; c < 8; c++)
                    *(uint4 *)(smem + kOffA2 + kb * kBlock + sw128_off(r, c)) =
                        make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
            }
            if (!__all_sync(0xffffffffu, ok)) break;
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive_first(bar(kBarA2));
            load_rec(i + 2, tid_next, rec);
            tid_next = task_of(own(i + 3));
        }
    } else if (warp >= 2) {
        /* ---- back warps: E2's epilogue and pooling ---- */
        const int q = warp & 3;
        const int h = (warp - 2 - kFrontWarps) >> 2;      /* states 4h .. 4h + 3 of the tile */
        const int unit = kHalfUnits * rank + q * 32 + lane;
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const float bias2 = b2[unit];
        /* lane k < 4 holds the tests of state k of tile i, loaded ahead as
           the front's records are */
        auto state_of = [&](int i) {
            return i < mine && lane < 4 ? (pair + i * pairs) * kStatesPerTile + 4 * h + lane : n;
        };
        auto task_of = [&](int s) -> int { return s < n ? (int)task[s] : -1; };
        auto tests_of = [&](int tid) { return tid < 0 ? 0 : min(task_T[tid], TP); };
        int T_cur = tests_of(task_of(state_of(0))), tid_next = task_of(state_of(1));
        for (int i = 0; i < mine; i++) {
            const int T_next = tests_of(tid_next);
            tid_next = task_of(state_of(i + 2));
            const bool ok = mbar_wait(bar(kBarE2 + kKB2 - 1), i & 1, abort_flag, status, 8);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_after();
            const int s0 = (pair + i * pairs) * kStatesPerTile + 4 * h;
            /* the four states' accumulators + bias, ReLU, bf16: D2 is drained
               before anything is summed */
            const uint32_t d2 = tmem + kUnits + lane_base + (uint32_t)(128 * h);
            uint32_t x[4][16];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                uint32_t acc[32];
                tmem_ld32(d2 + 32 * k, acc);
                if (k == 3) {
                    tc_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_first(bar(kBarFree2));
                }
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float2 u = add_f32x2(acc[2 * j], acc[2 * j + 1], bias2, bias2);
                    x[k][j] = relu_bf16x2(u.x, u.y);
                }
            }
            const float r_cur = 1.f / (float)(T_cur > 0 ? T_cur : 1);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                /* sum (fp32, tests in order, as k_pool) and max of this
                   lane's unit over the state's T columns, 8 tests at a time:
                   T is the warp's, so whole groups past it are skipped and
                   only the last one looks at each test */
                const int T = __shfl_sync(0xffffffffu, T_cur, k);
                const float r = __shfl_sync(0xffffffffu, r_cur, k);
                float v = 0.f;
                uint32_t m = 0u;              /* ReLU outputs are >= 0 */
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    if (8 * g >= T) break;
#pragma unroll
                    for (int j = 4 * g; j < 4 * g + 4; j++) {
                        if (8 * g + 8 > T)
                            x[k][j] &= (2 * j < T ? 0xFFFFu : 0u) | (2 * j + 1 < T ? 0xFFFF0000u : 0u);
                        v = add_bf16x2(v, x[k][j]);
                        m = max_bf16x2(m, x[k][j]);
                    }
                }
                if (s0 + k >= n) continue;
                m = max_bf16x2(m, m >> 16);
                __nv_bfloat16 *row = P + (size_t)(s0 + k) * kPoolCols + unit;
                row[0] = __float2bfloat16(quotient(v, T, r));
                reinterpret_cast<uint16_t *>(row)[kUnits] = (uint16_t)m;
            }
            T_cur = T_next;
        }
    }
    __syncwarp();
    tc_before();
    __syncthreads();
    cluster_sync();
    tc_after();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem)
                     : "memory");
}

/* ---- the training GEMM ------------------------------------------------------
 *
 * C[M,N] = A[M,K] . B[N,K]^T on tcgen05, both operands K-major bf16 in HBM,
 * FP32 accumulation in TMEM. One CTA per 128 x bn tile of C (bn <= 256, a
 * multiple of 16), grid.z splits K. Warp 0 (one thread) streams 64-column K
 * blocks of A (128 rows) and B (bn rows) by TMA with 128-byte swizzle
 * through a two-stage mbarrier ring; warp 1 owns TMEM and one thread issues
 * four tcgen05.mma (M=128, N=bn, K=16) per block; then all eight warps drain
 * the accumulators (warp w: TMEM lanes 32(w mod 4).. = tile rows, half w/4 of
 * the columns) with tcgen05.ld. Epilogue: with one K split, + bias, x (mask > 0) (the ReLU
 * derivative through a stored activation), ReLU, stored as bf16 or fp32;
 * with several, fp32 atomic adds into C (zeroed by the caller). Out-of-range
 * rows and columns of A and B are TMA zero fill; stores are bounds checked.
 * Every wait is bounded by the global timer; a wait that runs out sets the
 * abort flag and *status, each role leaves, and TMEM is freed. Two CTAs fit
 * an SM (96 KB of shared memory at bn = 256), so one CTA's epilogue overlaps
 * the other's loads and MMAs. The network's products are bound by their
 * bytes and this epilogue: 262,144 rows of 256, 67 us beside 39 of copy rate,
 * 90 with the mask beside 59; four warps, which found each 16-byte piece's
 * row by a division, took 94 and 142.
 *
 * mn_major: A and B are given K-row by K-row instead ([K][M] and [K][N],
 * M and N contiguous: the weight gradient dY^T . X reads dY [batch][out]
 * and X [batch][in] as stored), loaded as 64 x 64 boxes (64 K-rows of 64
 * elements along M or N) and described to the MMA as MN-major operands;
 * bn is then a multiple of 64. With kSums (mn_major only) four of the warps
 * that otherwise wait add up A's columns over the CTA's K rows from the same
 * stages, dY's column sums: the bias gradient without another pass over dY
 * (which took 37 us a layer of 262,144 rows; the product with the sums takes
 * 53 us where it took 52). A form of its own: the branches cost the others 5%. */
constexpr int kGRows = 128, kGBK = 64, kGStages = 2;
constexpr int kGABytes = kGRows * 128;              /* 16 KB per A stage */
constexpr int kGThreads = 256;
constexpr int kGSumWarps = 4;                       /* warps 2..5 */

template <bool kSums>
__global__ void __launch_bounds__(kGThreads, 2)
k_gemm_tc(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
          const float *__restrict__ bias, const __nv_bfloat16 *__restrict__ mask, int ldm,
          __nv_bfloat16 *__restrict__ Cb, float *__restrict__ Cf, int ldc, int M, int N,
          int kblocks, int kb_per_split, int bn, uint32_t idesc, uint32_t tmem_cols, int relu,
          int atomic_out, int stage_mode, int vec_atomic, int mn_major, float *part_db, int *status)
{
    extern __shared__ uint8_t gsmem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)gsmem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t b_bytes = (uint32_t)bn * 128u;
    const uint32_t sA = smem_u32(smem);
    const uint32_t sB = sA + kGStages * kGABytes;
    uint8_t *ctl = smem + kGStages * (kGABytes + b_bytes);
    const uint32_t sBar = smem_u32(ctl);
    uint32_t *tmem_slot = (uint32_t *)(ctl + 64);
    volatile int *abort_flag = (volatile int *)(ctl + 68);
    auto full = [&](int s) { return sBar + 8u * (uint32_t)s; };
    auto empty = [&](int s) { return sBar + 8u * (uint32_t)(kGStages + s); };
    const uint32_t done_bar = sBar + 8u * (uint32_t)(2 * kGStages);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * kGRows, n0 = blockIdx.x * bn;
    const int kb0 = blockIdx.z * kb_per_split;
    const int nk = min(kblocks, kb0 + kb_per_split) - kb0;

    /* the columns of A are summed once per row tile and K split */
    const bool sums = kSums && blockIdx.x == 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kGStages; s++) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), sums ? 1 + kGSumWarps : 1);
        }
        mbar_init(done_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)), "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0 && nk > 0) {
        /* producer */
        int i = 0;
        for (; i < nk; i++) {
            const int st = i % kGStages;
            const uint32_t ph = (uint32_t)(i / kGStages) & 1u;
            if (!mbar_wait(empty(st), ph ^ 1u, abort_flag, status, 11)) break;
            mbar_expect_tx(full(st), kGABytes + b_bytes);
            const int x = (kb0 + i) * kGBK;
            if (mn_major) {
                /* boxes of 64 K-rows x 64 columns, 8 KB each */
                for (int h = 0; h < kGRows / 64; h++)
                    tma_load_2d(sA + st * kGABytes + h * 8192, &map_a, full(st), m0 + 64 * h, x);
                for (int h = 0; h < bn / 64; h++)
                    tma_load_2d(sB + st * b_bytes + h * 8192, &map_b, full(st), n0 + 64 * h, x);
            } else {
                tma_load_2d(sA + st * kGABytes, &map_a, full(st), x, m0);
                tma_load_2d(sB + st * b_bytes, &map_b, full(st), x, n0);
            }
        }
        /* the copies this thread issued land before the CTA leaves */
        for (int j = i - 1; j >= 0 && j >= i - kGStages; j--) {
            const unsigned long long t0 = global_ns();
            while (!mbar_test(full(j % kGStages), (uint32_t)(j / kGStages) & 1u) &&
                   global_ns() - t0 < kWaitNs) {
            }
        }
    } else if (warp == 1 && lane == 0) {
        /* MMA issuer */
        for (int i = 0; i < nk; i++) {
            const int st = i % kGStages;
            const uint32_t ph = (uint32_t)(i / kGStages) & 1u;
            if (!mbar_wait(full(st), ph, abort_flag, status, 12)) break;
            tc_after();
            const uint32_t a0 = sA + st * kGABytes, b0 = sB + st * b_bytes;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                /* 16 K per MMA: 32 bytes along a K-major row, or two 8-row
                   groups (2 KB) of an MN-major box */
                const uint64_t da = mn_major ? sw128_mn_desc(a0 + 2048 * k) : sw128_desc(a0 + 32 * k);
                const uint64_t db = mn_major ? sw128_mn_desc(b0 + 2048 * k) : sw128_desc(b0 + 32 * k);
                const uint32_t acc = (i | k) != 0;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(idesc), "r"(acc)
                    : "memory");
            }
            mma_commit(empty(st));
        }
        /* arrives once every MMA above has completed (also after an abort);
           this thread waits for it, so TMEM is never freed under an MMA */
        mma_commit(done_bar);
        const unsigned long long t0 = global_ns();
        while (!mbar_test(done_bar, 0) && global_ns() - t0 < kWaitNs) {
        }
    }
    float col[8] = {};
    const int chunk = threadIdx.x & 15, slot = ((int)threadIdx.x - 64) >> 4;
    if (sums && warp >= 2 && warp < 2 + kGSumWarps) {
        /* a thread adds 8 columns (a 16-byte chunk of a row; 8 chunks of a
           64-column box's swizzled row) of every 8th K row */
        for (int i = 0; i < nk; i++) {
            const int st = i % kGStages;
            const bool ok = mbar_wait(full(st), (uint32_t)(i / kGStages) & 1u, abort_flag, status, 14);
            if (!__all_sync(0xFFFFFFFFu, ok)) break;
            const uint8_t *box = smem + st * kGABytes + (chunk >> 3) * 8192;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const uint4 v = *(const uint4 *)(box + sw128_off(slot + 8 * k, chunk & 7));
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    col[2 * j] += __uint_as_float(w[j] << 16);
                    col[2 * j + 1] += __uint_as_float(w[j] & 0xFFFF0000u);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty(st));
        }
    }
    __syncwarp();
    /* epilogue: all eight warps. The tile's bias goes to shared memory
       first (every thread takes part, so the barrier below is reached by
       all of them whatever the waits return). */
    float *sbias = (float *)(ctl + 256);
    for (int c = threadIdx.x; c < bn; c += kGThreads) sbias[c] = (bias && n0 + c < N) ? bias[n0 + c] : 0.f;
    bool ok = nk > 0 && mbar_wait(done_bar, 0, abort_flag, status, 13);
    ok = __all_sync(0xFFFFFFFFu, ok) && !*abort_flag;
    tc_after();
    __syncthreads();
    if (sums) {
        /* every stage is drained: the 8 row slots' sums meet there */
        float *ssum = (float *)smem;
        if (warp >= 2 && warp < 2 + kGSumWarps)
#pragma unroll
            for (int j = 0; j < 8; j++) ssum[slot * kGRows + 8 * chunk + j] = col[j];
        __syncthreads();
        if (ok && threadIdx.x < kGRows && m0 + (int)threadIdx.x < M) {
            float v = 0.f;
#pragma unroll
            for (int y = 0; y < 8; y++) v += ssum[y * kGRows + threadIdx.x];
            part_db[(size_t)blockIdx.z * M + m0 + threadIdx.x] = v;
        }
    }
    /* two warps share a TMEM lane quarter (32 rows), half of the columns each */
    const int quarter = warp & 3, half = (bn / 2 + 31) / 32 * 32;
    const int lo = warp < 4 ? 0 : min(half, bn), hi = warp < 4 ? min(half, bn) : bn;
    if (ok && stage_mode) {
        /* Staged: each warp drains its 32 rows of accumulators (+ bias,
           ReLU, rounding) into the drained stage buffers, a row of bn values
           at a stride of one row + 16 bytes (16-byte stores of eight lanes
           fall on distinct bank groups), then writes its rows to C in
           16-byte pieces, lanes along a row (coalesced), applying the mask
           on the way. stage_mode 1: bf16 C; 2: fp32 C (bn <= 112). */
        const int esz = stage_mode == 1 ? 2 : 4;
        const uint32_t S = (uint32_t)(bn * esz + 16);
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        uint8_t *rows = smem + (uint32_t)(quarter * 32) * S;
        uint8_t *myrow = rows + (uint32_t)lane * S;
        for (int c0 = lo; c0 < hi; c0 += 32) {
            uint32_t acc[32];
            tmem_ld32(tmem + lane_base + (uint32_t)c0, acc);
            if (stage_mode == 1) {
                uint32_t w[16];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float4 bv = *(const float4 *)(sbias + c0 + 4 * j);
                    const float2 u = add_f32x2(acc[4 * j], acc[4 * j + 1], bv.x, bv.y);
                    const float2 v = add_f32x2(acc[4 * j + 2], acc[4 * j + 3], bv.z, bv.w);
                    if (relu) {
                        w[2 * j] = relu_bf16x2(u.x, u.y);
                        w[2 * j + 1] = relu_bf16x2(v.x, v.y);
                    } else {
                        const __nv_bfloat162 hu = __floats2bfloat162_rn(u.x, u.y);
                        const __nv_bfloat162 hv = __floats2bfloat162_rn(v.x, v.y);
                        w[2 * j] = *reinterpret_cast<const uint32_t *>(&hu);
                        w[2 * j + 1] = *reinterpret_cast<const uint32_t *>(&hv);
                    }
                }
                /* the tile may end inside this group of 32 (bn = 16) */
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (c0 + 8 * k < hi)
                        *(uint4 *)(myrow + c0 * 2 + 16 * k) =
                            make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
            } else {
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    float v[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        v[q] = __uint_as_float(acc[4 * k + q]) + sbias[c0 + 4 * k + q];
                        if (relu) v[q] = fmaxf(v[q], 0.f);
                    }
                    if (c0 + 4 * k < hi)
                        *(float4 *)(myrow + c0 * 4 + 16 * k) = make_float4(v[0], v[1], v[2], v[3]);
                }
            }
        }
        __syncwarp();
        /* the warp's columns of its 32 rows in 16-byte pieces, a lane a piece
           and four at a time (their mask pieces all in flight); a lane's next
           piece is 32 further, its row and column follow without a division */
        const int per = 16 / esz;                 /* values per 16-byte piece */
        const int cpr = (hi - lo) / per;          /* pieces per row */
        const int dr = cpr ? 32 / cpr : 0, dc = cpr ? 32 - dr * cpr : 0;
        int r = cpr ? lane / cpr : 32, ch = cpr ? lane - r * cpr : 0;
        while (r < 32) {
            int rk[4], ck[4];
            uint4 mk[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                rk[k] = r;
                ck[k] = lo + ch * per;
                const int grow = m0 + quarter * 32 + r, gcol = n0 + ck[k];
                if (r >= 32 || grow >= M || gcol >= N) rk[k] = -1;
                else if (stage_mode == 1 && mask)
                    mk[k] = *(const uint4 *)(mask + (size_t)grow * ldm + gcol);
                ch += dc;
                r += dr;
                if (ch >= cpr) {
                    ch -= cpr;
                    r++;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (rk[k] < 0) continue;
                const size_t grow = (size_t)(m0 + quarter * 32 + rk[k]);
                const int gcol = n0 + ck[k];
                const uint8_t *src = rows + (uint32_t)rk[k] * S + ck[k] * esz;
                if (stage_mode == 1) {
                    uint4 v = *(const uint4 *)src;
                    if (mask) {
                        /* keep a value where its mask half is a positive bf16 */
                        auto keep = [](uint32_t m) {
                            return (__uint_as_float(m << 16) > 0.f ? 0x0000FFFFu : 0u) |
                                   (__uint_as_float(m & 0xFFFF0000u) > 0.f ? 0xFFFF0000u : 0u);
                        };
                        v.x &= keep(mk[k].x);
                        v.y &= keep(mk[k].y);
                        v.z &= keep(mk[k].z);
                        v.w &= keep(mk[k].w);
                    }
                    if (gcol + per <= N) {
                        *(uint4 *)(Cb + grow * ldc + gcol) = v;
                    } else {
                        const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int q = 0; q < 8; q++)
                            if (gcol + q < N)
                                reinterpret_cast<uint16_t *>(Cb)[grow * ldc + gcol + q] =
                                    (uint16_t)(w4[q >> 1] >> (16 * (q & 1)));
                    }
                } else {
                    const float4 v = *(const float4 *)src;
                    if (gcol + per <= N) {
                        *(float4 *)(Cf + grow * ldc + gcol) = v;
                    } else {
                        const float f4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (gcol + q < N) Cf[grow * ldc + gcol + q] = f4[q];
                    }
                }
            }
        }
    } else if (ok) {
        /* direct: split-K partial sums (fp32 adds, four at a time where
           aligned) or outputs the staged forms do not cover */
        const int row = m0 + quarter * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        for (int c0 = lo; c0 < hi; c0 += 32) {
            uint32_t acc[32];
            tmem_ld32(tmem + lane_base + (uint32_t)c0, acc);
            if (row >= M) continue;
            const int colb = n0 + c0;
            if (atomic_out == 2) {
                /* this K split's own slab: plain stores, summed later in
                   split order (deterministic) */
                float *dst = Cf + ((size_t)blockIdx.z * M + row) * ldc + colb;
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    if (vec_atomic && colb + j + 3 < N) {
                        *(float4 *)(dst + j) =
                            make_float4(__uint_as_float(acc[j]), __uint_as_float(acc[j + 1]),
                                        __uint_as_float(acc[j + 2]), __uint_as_float(acc[j + 3]));
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (colb + j + q < N) dst[j + q] = __uint_as_float(acc[j + q]);
                    }
                }
                continue;
            }
            if (atomic_out) {
                float *dst = Cf + (size_t)row * ldc + colb;
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    if (vec_atomic && colb + j + 3 < N) {
                        atomicAdd((float4 *)(dst + j),
                                  make_float4(__uint_as_float(acc[j]), __uint_as_float(acc[j + 1]),
                                              __uint_as_float(acc[j + 2]), __uint_as_float(acc[j + 3])));
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (colb + j + q < N) atomicAdd(dst + j + q, __uint_as_float(acc[j + q]));
                    }
                }
                continue;
            }
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const int c = colb + j;
                if (c >= N) continue;
                float v0 = __uint_as_float(acc[j]) + sbias[c0 + j];
                float v1 = __uint_as_float(acc[j + 1]) + sbias[c0 + j + 1];
                if (mask) {
                    const __nv_bfloat16 *mr = mask + (size_t)row * ldm + c;
                    if (!(__bfloat162float(mr[0]) > 0.f)) v0 = 0.f;
                    if (c + 1 < N && !(__bfloat162float(mr[1]) > 0.f)) v1 = 0.f;
                }
                if (relu) {
                    v0 = fmaxf(v0, 0.f);
                    v1 = fmaxf(v1, 0.f);
                }
                if (Cb) {
                    if (c + 1 < N)
                        *(__nv_bfloat162 *)(Cb + (size_t)row * ldc + c) = __floats2bfloat162_rn(v0, v1);
                    else
                        Cb[(size_t)row * ldc + c] = __float2bfloat16(v0);
                }
                if (Cf) {
                    Cf[(size_t)row * ldc + c] = v0;
                    if (c + 1 < N) Cf[(size_t)row * ldc + c + 1] = v1;
                }
            }
        }
    }
    tc_before();
    __syncthreads();
    tc_after();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(tmem_cols)
                     : "memory");
}

/* ---- the scoring trunk -------------------------------------------------------
 *
 * Z1 = relu(P . T1^T + b), Z2 = relu(Z1 . T2^T + b), logits = Z2 . H^T + b of
 * 128 pooled rows a tile in one kernel, a persistent CTA per SM; Z1 and Z2
 * stay in shared memory. Warp 0 streams P's blocks and the weights (370 KB a
 * tile, from L2) by TMA through a two-stage ring, a thread of warp 1 issues
 * the MMAs (M = 128; N = 256, 128, 16; the GEMM kernel's order of K blocks,
 * so its results), eight warps (two a TMEM lane quarter) are the epilogues.
 * The products run in the order T1(i + 1), T2(i), H(i - 1), so each
 * epilogue's work lies beside the others' products.
 *
 * Bound by the operands' way from L2, 670 KB a tile. As three launches of
 * k_gemm_tc Z1 and Z2 went through HBM: 131,072 rows 122 -> 64 us, and
 * 4,096 rows, mostly the three calls, 57 -> 21. */
constexpr int kTK1 = 9, kTK2 = 4, kTK3 = 2;           /* 64-column K blocks: 528, 256, 128 */
constexpr int kTStages = 2;
constexpr int kTStage = 3 * kBlock;                   /* A 16 KB, then B up to 32 KB */
constexpr int kTOffZ1 = kTStages * kTStage;           /* 64 KB */
constexpr int kTOffZ2 = kTOffZ1 + kTK2 * kBlock;      /* 32 KB */
constexpr int kTOffBias = kTOffZ2 + kTK3 * kBlock;    /* 256 + 128 + 16 fp32 */
constexpr int kTOffBar = kTOffBias + 400 * 4;
constexpr int kTSmem = kTOffBar + 256 + 1024;
constexpr int kTEpiWarps = 8, kTThreads = 64 + 32 * kTEpiWarps;
constexpr int kTFull = 0, kTEmpty = kTStages, kTD1 = 2 * kTStages, kTD2 = kTD1 + 1,
              kTD3 = kTD1 + 2, kTZ1 = kTD1 + 3, kTZ2 = kTD1 + 4, kTFree1 = kTD1 + 5,
              kTFree2 = kTD1 + 6, kTFree3 = kTD1 + 7, kTDrain = kTD1 + 8, kTBars = kTD1 + 9;
static_assert(kTSmem <= 227 * 1024 && kTOffBar % 8 == 0 && kTBars * 8 + 8 <= 256, "shared memory");
constexpr uint32_t kTColD2 = 256, kTColD3 = 384;      /* D1: columns 0..255 */

__device__ __forceinline__ void mma_one(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t idesc,
                                        uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__global__ void __launch_bounds__(kTThreads, 1)
k_trunk_tc(const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_w1,
           const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_w3,
           const float *__restrict__ b1, const float *__restrict__ b2,
           const float *__restrict__ b3, int n, float *__restrict__ logits, int *status)
{
    extern __shared__ uint8_t tsmem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)tsmem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem), sBar = sbase + kTOffBar;
    uint32_t *tmem_slot = (uint32_t *)(smem + kTOffBar + kTBars * 8);
    volatile int *abort_flag = (volatile int *)(smem + kTOffBar + kTBars * 8 + 4);
    float *bias = (float *)(smem + kTOffBias);
    auto bar = [&](int i) { return sBar + 8u * (uint32_t)i; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ntiles = (n + kRows - 1) / kRows;
    const int mine = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    auto row0 = [&](int i) { return ((int)blockIdx.x + i * (int)gridDim.x) * kRows; };

    if (threadIdx.x == 0) {
        for (int i = 0; i < kTBars; i++)
            mbar_init(bar(i), i >= kTZ1 && i <= kTFree2 ? kTEpiWarps : i == kTFree3 ? 4 : 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    for (int i = threadIdx.x; i < 400; i += kTThreads)
        bias[i] = i < 256 ? b1[i] : i < 384 ? b2[i - 256] : b3[i - 384];
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                         smem_u32(tmem_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        /* ---- TMA producer, in the order of the products ---- */
        if (lane == 0) {
            uint32_t j = 0;
            auto stage = [&](uint32_t bytes, uint32_t &st) {
                st = j % kTStages;
                if (!mbar_wait(bar(kTEmpty + st), ((j / kTStages) & 1u) ^ 1u, abort_flag, status, 21))
                    return false;
                mbar_expect_tx(bar(kTFull + st), bytes);
                j++;
                return true;
            };
            auto t1 = [&](int i) {
                for (int k = 0; k < kTK1; k++) {
                    uint32_t st;
                    if (!stage(kTStage, st)) return false;
                    tma_load_2d(sbase + st * kTStage, &map_p, bar(kTFull + st), 64 * k, row0(i));
                    tma_load_2d(sbase + st * kTStage + kBlock, &map_w1, bar(kTFull + st), 64 * k, 0);
                }
                return true;
            };
            auto weights = [&](const CUtensorMap *map, int blocks, uint32_t bytes) {
                for (int k = 0; k < blocks; k++) {
                    uint32_t st;
                    if (!stage(bytes, st)) return false;
                    tma_load_2d(sbase + st * kTStage + kBlock, map, bar(kTFull + st), 64 * k, 0);
                }
                return true;
            };
            bool ok = mine > 0 && t1(0);
            for (int i = 0; i <= mine && ok; i++) {
                if (i + 1 < mine) ok = t1(i + 1);
                if (ok && i < mine) ok = weights(&map_w2, kTK2, kBlock);
                if (ok && i > 0) ok = weights(&map_w3, kTK3, 16 * 128);
            }
            /* the copies this thread issued land before the CTA leaves */
            for (uint32_t back = 1; back <= kTStages && back <= j; back++) {
                const uint32_t last = j - back;
                const unsigned long long t0 = global_ns();
                while (!mbar_test(bar(kTFull + last % kTStages), (last / kTStages) & 1u) &&
                       global_ns() - t0 < kWaitNs) {
                }
            }
        }
    } else if (warp == 1) {
        /* ---- MMA issuer ---- */
        if (lane == 0) {
            uint32_t j = 0;
            auto wait = [&](int which, int tile, int code) {
                return mbar_wait(bar(which), tile & 1, abort_flag, status, code);
            };
            /* blocks of a product: A from the ring (z < 0) or from shared
               memory at offset z; the last block has `last` K steps */
            auto product = [&](int blocks, int last, int z, uint32_t col, int N, int done) {
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) |
                                       ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
                for (int kb = 0; kb < blocks; kb++, j++) {
                    const uint32_t st = j % kTStages;
                    if (!mbar_wait(bar(kTFull + st), (j / kTStages) & 1u, abort_flag, status, 22))
                        return false;
                    tc_after();
                    const uint32_t ring = sbase + st * kTStage;
                    const uint64_t da = sw128_desc(z < 0 ? ring : sbase + z + kb * kBlock);
                    const uint64_t db = sw128_desc(ring + kBlock);
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (kb + 1 < blocks || k < last)
                            mma_one(tmem + col, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                    mma_commit(bar(kTEmpty + st));
                }
                mma_commit(bar(done));
                return true;
            };
            auto t1 = [&](int i) {
                if (i && !wait(kTFree1, i - 1, 23)) return false;
                tc_after();
                return product(kTK1, 1, -1, 0, 256, kTD1);
            };
            bool ok = mine > 0 && t1(0);
            for (int i = 0; i <= mine && ok; i++) {
                if (i + 1 < mine) ok = t1(i + 1);
                if (ok && i < mine) {
                    ok = wait(kTZ1, i, 24) && (!i || wait(kTFree2, i - 1, 25));
                    tc_after();
                    ok = ok && product(kTK2, 4, kTOffZ1, kTColD2, 128, kTD2);
                }
                if (ok && i > 0) {
                    ok = wait(kTZ2, i - 1, 26) && (i < 2 || wait(kTFree3, i - 2, 27));
                    tc_after();
                    ok = ok && product(kTK3, 4, kTOffZ2, kTColD3, 16, kTD3);
                }
            }
            /* every MMA this thread issued has finished before TMEM is freed */
            mma_commit(bar(kTDrain));
            const unsigned long long t0 = global_ns();
            while (!mbar_test(bar(kTDrain), 0) && global_ns() - t0 < kWaitNs) {
            }
        }
    } else {
        /* ---- epilogues: two warps a lane quarter (32 rows), half of the
           columns each ---- */
        const int q = warp & 3, h = (warp - 2) >> 2;
        const int r = q * 32 + lane;
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        /* 32 columns of accumulators + bias, ReLU, bf16 */
        auto drain = [&](uint32_t col, const float *b, uint32_t *w) {
            uint32_t acc[32];
            tmem_ld32(tmem + lane_base + col, acc);
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const float4 bv = *(const float4 *)(b + 4 * c);
                const float2 u = add_f32x2(acc[4 * c], acc[4 * c + 1], bv.x, bv.y);
                const float2 v = add_f32x2(acc[4 * c + 2], acc[4 * c + 3], bv.z, bv.w);
                w[2 * c] = relu_bf16x2(u.x, u.y);
                w[2 * c + 1] = relu_bf16x2(v.x, v.y);
            }
        };
        /* a K block (64 columns) of the next product's operand */
        auto store = [&](int off, const uint32_t *w) {
#pragma unroll
            for (int c = 0; c < 8; c++)
                *(uint4 *)(smem + off + sw128_off(r, c)) =
                    make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
        };
        auto arrive = [&](int which) {
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(which));
        };
        auto wait = [&](int which, int tile, int code) {
            const bool done = mbar_wait(bar(which), tile & 1, abort_flag, status, code);
            return __all_sync(0xffffffffu, done) != 0;
        };
        for (int i = 0; i < mine + 2 && mine; i++) {
            if (i < mine) {
                /* T1(i) into Z1, once T2(i - 1) has read it */
                if (!wait(kTD1, i, 28)) break;
                tc_after();
                uint32_t w[64];
#pragma unroll
                for (int g = 0; g < 4; g++)
                    drain((uint32_t)(128 * h + 32 * g), bias + 128 * h + 32 * g, w + 16 * g);
                tc_before();
                arrive(kTFree1);
                if (i && !wait(kTD2, i - 1, 29)) break;
#pragma unroll
                for (int k = 0; k < 2; k++) store(kTOffZ1 + (2 * h + k) * kBlock, w + 32 * k);
                fence_async_smem();
                arrive(kTZ1);
            }
            if (i >= 1 && i <= mine) {
                /* T2(i - 1) into Z2, once H(i - 2) has read it */
                if (!wait(kTD2, i - 1, 30)) break;
                tc_after();
                uint32_t w[32];
#pragma unroll
                for (int g = 0; g < 2; g++)
                    drain(kTColD2 + 64 * h + 32 * g, bias + 256 + 64 * h + 32 * g, w + 16 * g);
                tc_before();
                arrive(kTFree2);
                if (i >= 2 && !wait(kTD3, i - 2, 31)) break;
                store(kTOffZ2 + h * kBlock, w);
                fence_async_smem();
                arrive(kTZ2);
            }
            if (i >= 2 && h == 0) {
                /* H(i - 2): the logits, a row a lane */
                if (!wait(kTD3, i - 2, 32)) break;
                tc_after();
                uint32_t acc[32];
                tmem_ld32(tmem + lane_base + kTColD3, acc);
                tc_before();
                arrive(kTFree3);
                const int row = row0(i - 2) + r;
                if (row < n)
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const float4 b = *(const float4 *)(bias + 384 + 4 * c);
                        *(float4 *)(logits + (size_t)row * 16 + 4 * c) =
                            make_float4(__uint_as_float(acc[4 * c]) + b.x,
                                        __uint_as_float(acc[4 * c + 1]) + b.y,
                                        __uint_as_float(acc[4 * c + 2]) + b.z,
                                        __uint_as_float(acc[4 * c + 3]) + b.w);
                    }
            }
        }
    }
    __syncwarp();
    tc_before();
    __syncthreads();
    tc_after();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem)
                     : "memory");
}


typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                             &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    });
    return fn;
}

/* Tensor map of a row-major [256][K] bf16 weight, boxes of 64 columns x `units`
   rows, 128B swizzle. */
bool weight_map(CUtensorMap *m, const void *W, int K, int units)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)kUnits};
    cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)units};
    cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(W), dims, strides, box,
              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

/* Tensor map of a row-major [rows][cols] bf16 matrix (row stride ld
   elements), boxes of 64 columns x box_rows rows, 128-byte swizzle. */
bool tile_map(CUtensorMap *m, const void *ptr, int rows, int cols, int ld, int box_rows)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box,
              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

/* Allow a kernel `bytes` of dynamic shared memory on the current device. */
template <class Kernel>
bool allow_smem(pcagb::OncePerDevice &once, Kernel *kernel, int bytes)
{
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && once.run(dev, [&] {
        const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             bytes) == cudaSuccess;
        if (!ok) cudaGetLastError();   /* reported here, not by the next launch */
        return ok;
    });
}

constexpr int kGSmemMost = kGStages * (kGABytes + 256 * 128) + 256 + 2048;
pcagb::OncePerDevice g_gemm_smem, g_gemm_sums_smem;

}  // namespace

/* C[M,N] = A[M,K] . B[N,K]^T on tcgen05 (k_gemm_tc): bias[N] added, then
 * columns where mask[M][N] (bf16, leading dimension ldm) is not positive
 * zeroed, then ReLU, into Cb (bf16) and/or Cf (fp32), leading dimension ldc.
 * splits > 1 divides K among CTAs that add fp32 partial sums into Cf (zeroed
 * by the caller; no bias, mask, ReLU or Cb then). A and B: leading
 * dimensions multiples of 8 elements, 16-byte aligned. *status gets a
 * nonzero code if a barrier wait ran out (the result is then void). */
extern "C" int pcagb_vnet_gemm_tc(const void *A, int lda, const void *B, int ldb,
                                  const float *bias, const void *mask, int ldm, void *Cb,
                                  float *Cf, int ldc, int M, int N, int K, int relu, int splits,
                                  int *status, void *stream)
{
    if (M <= 0 || N <= 0 || K <= 0) return PCAGB_OK;
    if (!A || !B || !status || (!Cb && !Cf) || (lda & 7) || (ldb & 7) || lda < K || ldb < K ||
        ((uintptr_t)A & 15) || ((uintptr_t)B & 15) || splits < 1 ||
        (splits > 1 && (!Cf || Cb || bias || mask || relu)))
        return PCAGB_EINVAL;
    const int bn = N > 256 ? 256 : (N + 15) / 16 * 16;
    uint32_t tcols = 32;
    while (tcols < (uint32_t)bn) tcols <<= 1;
    CUtensorMap ma, mb;
    if (!tile_map(&ma, A, M, K, lda, kGRows) || !tile_map(&mb, B, N, K, ldb, bn))
        return PCAGB_ECUDA;
    const int kblocks = (K + kGBK - 1) / kGBK;
    if (splits > kblocks) splits = kblocks;
    const int per = (kblocks + splits - 1) / splits;
    splits = (kblocks + per - 1) / per;
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) |
                           ((uint32_t)(kGRows >> 4) << 24);
    /* stage buffers, then 256 bytes of barriers and flags, the tile's bias
       (bn floats), 1 KB of alignment slack */
    const int smem = kGStages * (kGABytes + bn * 128) + 256 + 1024 + 1024;
    /* the epilogue: staged through shared memory and stored in 16-byte
       pieces where the output's alignment allows */
    int stage_mode = 0;
    if (splits == 1 && Cb && !Cf && ldc % 8 == 0 && !((uintptr_t)Cb & 15) &&
        (!mask || (ldm % 8 == 0 && !((uintptr_t)mask & 15))))
        stage_mode = 1;
    else if (splits == 1 && Cf && !Cb && !mask && bn <= 112 && ldc % 4 == 0 &&
             !((uintptr_t)Cf & 15))
        stage_mode = 2;
    const int vec_atomic = splits > 1 && ldc % 4 == 0 && !((uintptr_t)Cf & 15);
    if (!allow_smem(g_gemm_smem, k_gemm_tc<false>, kGSmemMost)) return PCAGB_ECUDA;
    dim3 grid((N + bn - 1) / bn, (M + kGRows - 1) / kGRows, splits);
    k_gemm_tc<false><<<grid, kGThreads, smem, (cudaStream_t)stream>>>(
        ma, mb, bias, (const __nv_bfloat16 *)mask, ldm, (__nv_bfloat16 *)Cb, Cf, ldc, M, N,
        kblocks, per, bn, idesc, tcols, relu, splits > 1, stage_mode, vec_atomic, 0, nullptr, status);
    return cudaGetLastError() == cudaSuccess ? PCAGB_OK : PCAGB_ECUDA;
}

/* Tensor map of a [krows][cols] bf16 matrix (row stride ld elements) read
   as an MN-major operand: boxes of 64 columns x 64 rows, 128-byte swizzle. */
bool tile_map_mn(CUtensorMap *m, const void *ptr, int krows, int cols, int ld)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)krows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {64, 64};
    cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box,
              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

/* C[i] += the `splits` slabs' values at i, in slab order, and the same for
 * db from part_db (count_db values; 0: none): a thread per value, 16 slabs'
 * loads in flight before they are added (one after the other a value waits
 * for up to 152 loads in turn: 9 to 19 us a layer, so 8 to 12). */
__global__ void k_split_sum(const float *part, int splits, size_t count, float *C,
                            const float *part_db, size_t count_db, float *db)
{
    for (size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x; at < count + count_db;
         at += (size_t)gridDim.x * blockDim.x) {
        const bool first = at < count;
        const size_t i = first ? at : at - count, n = first ? count : count_db;
        const float *src = (first ? part : part_db) + i;
        float v = 0.f;
        int z = 0;
        for (; z + 16 <= splits; z += 16) {
            float p[16];
#pragma unroll
            for (int k = 0; k < 16; k++) p[k] = src[(size_t)(z + k) * n];
#pragma unroll
            for (int k = 0; k < 16; k++) v += p[k];
        }
        for (; z < splits; z++) v += src[(size_t)z * n];
        (first ? C : db)[i] += v;
    }
}

/* The number of K splits pcagb_vnet_wgrad_tc uses for this shape when asked
 * for `splits` (its partial buffer holds that many [M][ldc] slabs). */
extern "C" int pcagb_vnet_wgrad_splits(int K, int splits)
{
    const int kblocks = (K + kGBK - 1) / kGBK;
    if (splits < 1) splits = 1;
    if (splits > kblocks) splits = kblocks;
    const int per = (kblocks + splits - 1) / splits;
    return (kblocks + per - 1) / per;
}

/* Weight gradient on tcgen05 without transposes: C[M][N] += dY^T . X over
 * K rows, dY [K][M] (leading dimension ldy) and X [K][N] (ldx) read as
 * stored (MN-major operands), with the K rows in `splits` ranges. With
 * `part` (pcagb_vnet_wgrad_splits(K, splits) slabs of M x ldc floats) each
 * range writes its own slab and the slabs are added into C in range order,
 * so the result is the same on every run; without it the ranges' fp32 sums
 * are added into C atomically. C is zeroed by the caller (leading dimension
 * ldc). ldy and ldx are multiples of 8 elements, dY and X 16-byte aligned. */
static int wgrad(const void *dY, int ldy, const void *X, int ldx, float *C, int ldc, int M, int N,
                 int K, int splits, float *part, float *db, float *part_db, int *status,
                 void *stream)
{
    if (M <= 0 || N <= 0 || K <= 0) return PCAGB_OK;
    if (!dY || !X || !C || !status || (ldy & 7) || (ldx & 7) || ldy < M || ldx < N ||
        ldc < N || ((uintptr_t)dY & 15) || ((uintptr_t)X & 15) || splits < 1)
        return PCAGB_EINVAL;
    const int bn = N > 192 ? 256 : (N + 63) / 64 * 64;
    uint32_t tcols = 32;
    while (tcols < (uint32_t)bn) tcols <<= 1;
    CUtensorMap ma, mb;
    if (!tile_map_mn(&ma, dY, K, M, ldy) || !tile_map_mn(&mb, X, K, N, ldx)) return PCAGB_ECUDA;
    const int kblocks = (K + kGBK - 1) / kGBK;
    if (splits > kblocks) splits = kblocks;
    const int per = (kblocks + splits - 1) / splits;
    splits = (kblocks + per - 1) / per;
    /* bits 15 and 16: A and B MN-major */
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                           ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(kGRows >> 4) << 24);
    const int smem = kGStages * (kGABytes + bn * 128) + 256 + 1024 + 1024;
    if (!(part_db ? allow_smem(g_gemm_sums_smem, k_gemm_tc<true>, kGSmemMost)
                  : allow_smem(g_gemm_smem, k_gemm_tc<false>, kGSmemMost)))
        return PCAGB_ECUDA;
    float *out = part ? part : C;
    const int vec_atomic = ldc % 4 == 0 && !((uintptr_t)out & 15);
    dim3 grid((N + bn - 1) / bn, (M + kGRows - 1) / kGRows, splits);
    (part_db ? k_gemm_tc<true> : k_gemm_tc<false>)<<<grid, kGThreads, smem, (cudaStream_t)stream>>>(
        ma, mb, nullptr, nullptr, 0, nullptr, out, ldc, M, N, kblocks, per, bn, idesc, tcols, 0,
        part ? 2 : 1, 0, vec_atomic, 1, part_db, status);
    if (cudaGetLastError() != cudaSuccess) return PCAGB_ECUDA;
    if (part) {
        const size_t count = (size_t)M * ldc;
        const size_t count_db = part_db ? (size_t)M : 0;
        const unsigned blocks = (unsigned)std::min<size_t>((count + count_db + 63) / 64, 4096);
        k_split_sum<<<blocks, 64, 0, (cudaStream_t)stream>>>(part, splits, count, C, part_db,
                                                             count_db, db);
        if (cudaGetLastError() != cudaSuccess) return PCAGB_ECUDA;
    }
    return PCAGB_OK;
}

extern "C" int pcagb_vnet_wgrad_tc(const void *dY, int ldy, const void *X, int ldx, float *C,
                                   int ldc, int M, int N, int K, int splits, float *part,
                                   int *status, void *stream)
{
    return wgrad(dY, ldy, X, ldx, C, ldc, M, N, K, splits, part, nullptr, nullptr, status, stream);
}

/* The same with the bias gradient: db[M] += dY's column sums. part and
 * part_db (pcagb_vnet_wgrad_splits(K, splits) slabs of M floats) are needed. */
extern "C" int pcagb_vnet_wgrad_bias_tc(const void *dY, int ldy, const void *X, int ldx, float *C,
                                        int ldc, int M, int N, int K, int splits, float *part,
                                        float *db, float *part_db, int *status, void *stream)
{
    if (M > 0 && N > 0 && K > 0 && (!part || !db || !part_db)) return PCAGB_EINVAL;
    return wgrad(dY, ldy, X, ldx, C, ldc, M, N, K, splits, part, db, part_db, status, stream);
}


extern "C" int pcagb_vnet_encode_pool_tc(const void *W1, const float *b1, const void *W2,
                                         const float *b2, const uint16_t *regs,
                                         const uint8_t *flags, const uint8_t *live,
                                         const uint16_t *task, const uint8_t *depth, int TP, int n,
                                         const uint16_t *task_io, const int32_t *task_T, void *P,
                                         int *status, void *stream)
{
    if (n <= 0) return PCAGB_OK;
    if ((TP != 16 && TP != 32) || !W1 || !W2 || !b1 || !b2 || !P || !status ||
        ((uintptr_t)W1 & 15) || ((uintptr_t)W2 & 15))
        return PCAGB_EINVAL;
    CUtensorMap m1, m2;
    if (!weight_map(&m1, W1, kFeat, kHalfUnits / 2) || !weight_map(&m2, W2, kUnits, kHalfUnits)) return PCAGB_ECUDA;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return PCAGB_ECUDA;
    static pcagb::OncePerDevice smem;
    if (!allow_smem(smem, k_encode_pool_tc, kSmemBytes)) return PCAGB_ECUDA;
    const int ntiles = (n + kStatesPerTile - 1) / kStatesPerTile;
    const int pairs = ntiles < sms / 2 ? ntiles : sms / 2;
    k_encode_pool_tc<<<2 * pairs, kThreads, kSmemBytes, (cudaStream_t)stream>>>(
        m1, m2, b1, b2, regs, flags, live, task, depth, TP, n, task_io, task_T,
        (__nv_bfloat16 *)P, status);
    return cudaGetLastError() == cudaSuccess ? PCAGB_OK : PCAGB_ECUDA;
}

/* Logits [n][16] (fp32) of pooled rows P [n][528] through the trunk: T1 [256]
 * [528], T2 [128][256], H [16][128] bf16, row-major and contiguous. P, the
 * weights and the logits are 16-byte aligned. *status as in the other
 * tcgen05 launches. */
extern "C" int pcagb_vnet_trunk_tc(const void *P, int n, const void *T1, const float *b1,
                                   const void *T2, const float *b2, const void *H, const float *b3,
                                   float *logits, int *status, void *stream)
{
    if (n <= 0) return PCAGB_OK;
    if (!P || !T1 || !T2 || !H || !b1 || !b2 || !b3 || !logits || !status ||
        (((uintptr_t)P | (uintptr_t)T1 | (uintptr_t)T2 | (uintptr_t)H | (uintptr_t)logits) & 15))
        return PCAGB_EINVAL;
    CUtensorMap mp, m1, m2, m3;
    if (!tile_map(&mp, P, n, kPoolCols, kPoolCols, kRows) ||
        !tile_map(&m1, T1, 256, kPoolCols, kPoolCols, 256) ||
        !tile_map(&m2, T2, 128, 256, 256, 128) || !tile_map(&m3, H, 16, 128, 128, 16))
        return PCAGB_ECUDA;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return PCAGB_ECUDA;
    static pcagb::OncePerDevice smem;
    if (!allow_smem(smem, k_trunk_tc, kTSmem)) return PCAGB_ECUDA;
    const int ntiles = (n + kRows - 1) / kRows;
    k_trunk_tc<<<ntiles < sms ? ntiles : sms, kTThreads, kTSmem, (cudaStream_t)stream>>>(
        mp, m1, m2, m3, b1, b2, b3, n, logits, status);
    return cudaGetLastError() == cudaSuccess ? PCAGB_OK : PCAGB_ECUDA;
}
