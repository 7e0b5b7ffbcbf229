// Batched prompt processing: the positions of a prompt go through every layer up to 256 at a time, so a weight byte
// is read from HBM once per 256 tokens instead of once per token, and the dot products run on the tensor cores.
//
// The reference has no such path: its run loop pushes every prompt token through the decode step
// (Run.java:623-637).  What is computed per position is the decode step's arithmetic (Run.java:418-508): the
// same RMSNorm, the same 24-bit fixed-point form of the activations (one power-of-two scale per quantisation
// group, three balanced signed byte limbs), exact integer sums of u8 weights x s8 limbs, (min, scale) of the
// weight group applied in FP32 -- only the order of the FP32 additions over the groups of a row differs from
// the decode kernels, so prompt positions agree with them to rounding, not bit for bit.
//
// Kernels:
//   pf_embed_kernel     rows of the embedding table for the chunk's tokens
//   pf_limbs_kernel     activations -> limbs [3 x 64 rows][K] (the B operand) per block of 64 tokens + per (group,
//                       token) unit and sum; input is RMSNorm(x) * w, the attention output, or SwiGLU(h1, h3)
//   pf_gemm_kernel      C[64 tokens][rows] (+)= W[rows][K] x limbs: TMA (cp.async.bulk.tensor) feeds 128-byte-
//                       swizzled tiles to tcgen05.mma kind::i8 (u8 x s8 -> s32, M 128, N 3 x tokens, K 32), one
//                       accumulator per quantisation group in tensor memory, double-buffered; eight epilogue warps
//                       read it back (tcgen05.ld), scale in FP32 and keep the row sums in registers
//   pf_rope_kv_kernel   RoPE on q and k, rows of the K/V cache (ApplyRope.java:61-92, Run.java:443-455)
//   pf_attention_kernel causal attention of the chunk's queries over the cache: FP32 operands in three bf16 pieces on
//                       the tensor cores, online softmax in FP32

#include "l2j_device.cuh"
#include "l2j_internal.h"

#include <cuda.h>

#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#define PF_DS_WAIT_TIMEOUT 0x1u   // L2J_DS_WAIT_TIMEOUT of the public header

namespace l2j {

namespace {

constexpr int kT = kPrefillTokens;          // tokens per block of the B operand
constexpr int kTB = 4;                      // token blocks per chunk of a prompt.  A matrix launch costs about 9 us beside its
                                            // tiles (set-up, first copies, drain) and there are nine launches per layer and
                                            // chunk: with four blocks instead of one, 3840 tokens through 16 layers of the
                                            // 7B shape take 144 instead of 214 ms
constexpr int kN = 3 * kT;                  // columns of the B operand: three limbs per token
constexpr int kTileM = 128;                 // weight rows per tile
constexpr int kGemmThreads = 384;          // A producer, two issue warps, B producer, eight epilogue warps
constexpr int kEpiWarps = 8;                // warps 4..11: quarter of tensor memory = warp % 4, half of the tokens = (warp - 4) / 4
constexpr int kABytes = kTileM * 128;       // the A part of a stage: 128 rows of 128 bytes
constexpr int kMaxParts = 12;               // parts a row sum (or a query's keys) may be dealt into
constexpr int kWideParts = 3;               // at most this many parts for the wide outputs (W1/W3): their sums are read back
constexpr int kAccCols = 256;               // column distance of the two accumulators of the classifier in tensor memory
constexpr int kTmemCols = 512;
constexpr int kMaxDim = 16384;              // longest row of a matrix

// ---- tcgen05 / TMA wrappers ----------------------------------------------------------------------------------

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
                 : "memory");
}

__device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar, uint64_t policy)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "l"(policy)
        : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t smem_result, uint32_t cols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(cols) : "memory");
}

__device__ __forceinline__ void tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

__device__ __forceinline__ void tc_fence_before()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[smem] x B[smem], u8 x s8 -> s32
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// The barrier gets one arrival when every tcgen05 operation this thread has issued so far is complete.
__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *r)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld_wait()
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes, 128-byte swizzled (what the TMA
// writes with CU_TENSOR_MAP_SWIZZLE_128B): groups of 8 rows are 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr)
{
    uint64_t d = (uint64_t)((addr >> 4) & 0x3fffu);
    d |= (uint64_t)1 << 16;                 // leading byte offset (not used by swizzled K-major layouts)
    d |= (uint64_t)(1024 >> 4) << 32;       // stride byte offset
    d |= (uint64_t)1 << 46;                 // descriptor version of this architecture
    d |= (uint64_t)2 << 61;                 // 128-byte swizzle
    return d;
}

// The matrix kernel for blocks of TT tokens.  A call of few tokens (a step of a few sequences, a short prompt) takes the
// smallest that holds them: the tensor cores, the epilogue and the activation tiles cost as much for a token that does not
// exist, and what they leave free goes into a deeper ring and more accumulators.
template <int TT>
struct GemmCfg {
    static constexpr int kCols = 3 * TT;                       // columns of the B operand
    static constexpr int kStageBytes = kABytes + kCols * 128;
    // Ring depth, known at compile time: the two single-lane issue loops are on the critical path (a run-time depth, i.e. a
    // division per stage, costs 15 %).  One stage = half a quantisation group (K = 128) of A and B.
    static constexpr int kStages = TT <= 16 ? 8 : 4;
    static constexpr int kPairs = kStages / 2;                 // groups in the ring
    static constexpr int kAccs = TT <= 16 ? 8 : (TT <= 32 ? 4 : 2);
    static constexpr int kAccDist = 512 / kAccs;               // columns between two accumulators in tensor memory
    static constexpr int kHalf = TT / 2;                       // tokens per epilogue thread
    static constexpr int kChunk = kHalf % 16 ? 8 : 16;         // of them, taken from tensor memory at a time
    // The epilogue's count of groups.  At 64 tokens it has 64 bits: with 32 the compiler spills 40 / 124 bytes (stores / loads) there
    // instead of 4 / 20; 3840 tokens through 16 layers of the 7B shape 78.4 -> 77.6 ms.
    using Count = std::conditional_t<(TT > 48), long, unsigned int>;
    // c s32, a u8, b s8, both K-major, M 128
    static constexpr uint32_t kIdesc = (2u << 4) | (0u << 7) | (1u << 10) | ((uint32_t)(kCols >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
    static constexpr size_t smem(int groups) { return (size_t)kStages * kStageBytes + (size_t)groups * TT * sizeof(float2) + 1024; }
    // The two issue lanes take the groups in turn.  A pair of stages (an accumulator) must always come back to the same lane:
    // a lane that waits for a phase whose predecessor it has not seen itself may pass on the one before that.
    static_assert(kPairs % 2 == 0 && kAccs % 2 == 0, "a lane owns its stages and accumulators");
    static_assert(kCols % 16 == 0 && kCols <= kAccDist && kHalf % kChunk == 0, "shape of the instruction and of its accumulators");
    static_assert(kStages * kStageBytes + (kMaxDim / 256) * TT * 8 + 1024 <= 227 * 1024, "what a block may have");
};

// Bounded wait that also ends when another role of the block has given up.
__device__ __forceinline__ bool pf_wait(uint32_t bar, uint32_t parity, volatile int *give_up, long long limit)
{
    if (mbar_try_wait(bar, parity))
        return true;
    const long long c0 = sm_clock();
    for (;;) {
        if (mbar_try_wait(bar, parity))
            return true;
        if (*give_up != 0 || sm_clock() - c0 > limit) {
            *give_up = 1;
            return false;
        }
    }
}

__device__ __forceinline__ int dp4a_ones(uint32_t limbs, int acc)
{
    int r;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(0x01010101u), "r"(limbs), "r"(acc));
    return r;
}

}  // namespace

// ---------------------------------------------------------------------------------------------------------------
// GEMM
// ---------------------------------------------------------------------------------------------------------------

struct PfGemmSeg {
    const float2 *hdr;   // (min, scale) of group g of row r at hdr[r * groups + g]
    int rows;            // multiple of 128
    int col0;            // first output column of the segment
};

struct PfGemmParams {
    PfGemmSeg seg[3];
    int nseg;
    int groups;          // K / 256
    int tblocks;         // blocks of 64 tokens; the grid is a multiple of it, so a block's items are of one token block
    const float2 *ux;    // [tblocks][groups][64]: (value of one unit of the integer sums, sum of the fixed-point activations)
    const float *ssq;    // [tblocks][nssq][64] partial sums of squares of the input rows (RMSNorm in front), or nullptr
    int nssq;
    int n;               // elements per input row
    float *out;          // [ksplit][64 * tblocks][ldc]
    int ldc;
    int ksplit;          // the groups of a row are dealt to this many blocks; part z goes to out + z * 64 * tblocks * ldc
    int nvalid;          // tokens of the chunk that exist
    int timeout_us;
    unsigned int *status;
};

// 512: no more than 128 registers per thread, so that blocks of the kernels in front and behind fit on the SM beside it
template <int TT>
__global__ void __launch_bounds__(512, 1)
pf_gemm_kernel(const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_a1,
               const __grid_constant__ CUtensorMap map_a2, const __grid_constant__ CUtensorMap map_b, const PfGemmParams p)
{
    extern __shared__ unsigned char pf_smem_raw[];
    using C = GemmCfg<TT>;
    constexpr int kStages = C::kStages, kStageBytes = C::kStageBytes, kAccs = C::kAccs;
    __shared__ __align__(8) unsigned long long s_bar[2 * kStages + 2 * kAccs + 2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_give_up;
    __shared__ float s_ss[TT];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(pf_smem_raw) + 1023u) & ~1023u;            // swizzled tiles want 1024-byte alignment
    unsigned char *gen = pf_smem_raw + (base - smem_u32(pf_smem_raw));
    float2 *s_ux = reinterpret_cast<float2 *>(gen + (size_t)kStages * kStageBytes);
    const uint32_t bar_full = smem_u32(&s_bar[0]), bar_empty = smem_u32(&s_bar[kStages]);
    const uint32_t bar_acc_full = smem_u32(&s_bar[2 * kStages]), bar_acc_empty = smem_u32(&s_bar[2 * kStages + kAccs]);
    const uint32_t bar_fin = smem_u32(&s_bar[2 * kStages + 2 * kAccs]);
    const long long limit = 2000ll * (long long)p.timeout_us;

    int ntiles = 0;
    for (int s = 0; s < p.nseg; ++s)
        ntiles += p.seg[s].rows / kTileM;
    ntiles *= p.ksplit;                       // work items of this token block: (tile, part of the groups)
    const int G = p.groups;
    // blocks next to each other work on the same weights for different tokens: L2 serves all but the first
    const int tb = (int)blockIdx.x % p.tblocks, first = (int)blockIdx.x / p.tblocks, stride = (int)gridDim.x / p.tblocks;
    const int gper = (G + p.ksplit - 1) / p.ksplit;

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(bar_full + 8 * s, 2);            // both producers
            mbar_init(bar_empty + 8 * s, 1);
        }
        for (int b = 0; b < kAccs; ++b) {
            mbar_init(bar_acc_full + 8 * b, 1);
            mbar_init(bar_acc_empty + 8 * b, kEpiWarps);
        }
        mbar_init(bar_fin, 1);
        mbar_init(bar_fin + 8, 1);
        mbar_fence_init();
        s_give_up = 0;
    }
    auto tile_map = [&](int tile, int &m0) {
        int sg = 0;
        m0 = (tile / p.ksplit) * kTileM;
        while (m0 >= p.seg[sg].rows) {
            m0 -= p.seg[sg].rows;
            ++sg;
        }
        return sg == 0 ? &map_a0 : (sg == 1 ? &map_a1 : &map_a2);
    };
    pdl_launch_dependents();
    // The weights do not depend on the kernel in front: the first stages' tiles are on their way while it still runs.
    // Tensor memory is taken behind the wait only: nothing may hold it that waits for another kernel.
    int primed = 0;
    if (tid == 0 && first < ntiles) {
        int m0;
        const CUtensorMap *ma = tile_map(first, m0);
        const int g0 = (first % p.ksplit) * gper, g1 = min(G, g0 + gper);
        primed = max(0, min(kStages, 2 * (g1 - g0)));
        for (int s = 0; s < primed; ++s) {
            mbar_arrive_expect_tx(bar_full + 8 * s, kABytes);
            tma_load_2d_hint(base + (uint32_t)s * kStageBytes, ma, (2 * g0 + s) * 128, m0, bar_full + 8 * s, policy_evict_first());
        }
    }
    pdl_wait();
    if (warp == 1) {
        tmem_alloc(smem_u32(&s_tmem), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    volatile int *give_up = &s_give_up;

    if (warp == 0 || warp == 3) {
        // ---- producers: one lane feeds the weights to the ring, one the activations.  A wait and the issue of a copy take a
        // few hundred cycles, and a stage is used up in 500: one lane for both was as slow as everything else together.
        const bool weights = warp == 0;
        if (lane == 0) {
            const uint64_t pol = policy_evict_first();
            int it = 0, s = 0;
            uint32_t ph = 1;
            for (int tile = first; tile < ntiles && !*give_up; tile += stride) {
                int m0;
                const CUtensorMap *ma = tile_map(tile, m0);
                const int g0 = (tile % p.ksplit) * gper, g1 = min(G, g0 + gper);
                for (int hs = 2 * g0; hs < 2 * g1; ++hs, ++it) {   // half groups
                    const uint32_t st = base + (uint32_t)s * kStageBytes;
                    if (!weights || it >= primed) {
                        if (!pf_wait(bar_empty + 8 * s, ph, give_up, limit))
                            break;
                        mbar_arrive_expect_tx(bar_full + 8 * s, weights ? kABytes : C::kCols * 128);
                        if (weights)
                            tma_load_2d_hint(st, ma, hs * 128, m0, bar_full + 8 * s, pol);
                        else
                            tma_load_2d(st + kABytes, &map_b, hs * 128, tb * C::kCols, bar_full + 8 * s);
                    }
                    if (++s == kStages) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (*give_up) {
                // copies that nobody consumed must land before the block's shared memory goes away
                for (int i = 0; i < kStages; ++i)
                    for (uint32_t q = 0; q < 2; ++q) {
                        const long long c0 = sm_clock();
                        while (!mbar_try_wait(bar_full + 8 * i, q) && sm_clock() - c0 < limit) {
                        }
                    }
            }
        }
    } else if (warp <= 2) {
        // ---- tensor-core issue: one lane of each of two warps, which take the groups (and the accumulators) in turn.  The
        // issue of a group's eight instructions takes as long as the tensor cores need for them (900 cycles), and the waits,
        // fences and commits around it as long again: with one lane the tensor cores idled through the latter.  With this
        // and two producer lanes 256 tokens through 16 layers of the 7B shape take 3.83 instead of 4.17 ms.
        if (lane == 0) {
            const int b = warp - 1;
            int mine = 0;                        // groups of the block that are this lane's: every second one
            for (int tile = first; tile < ntiles; tile += stride) {
                const int g0 = (tile % p.ksplit) * gper;
                mine += max(0, min(G, g0 + gper) - g0);
            }
            mine = (mine + 1 - b) / 2;
            bool ok = true;
            int pair = b % C::kPairs, acc = b % kAccs;             // of the lane's next group: two stages of the ring, an accumulator
            uint32_t ph = (uint32_t)(b / C::kPairs) & 1u, pha = (uint32_t)(b / kAccs) & 1u;
            for (; mine > 0 && ok; --mine) {
                const uint32_t d = tmem + (uint32_t)(acc * C::kAccDist), ta = base + (uint32_t)(2 * pair) * kStageBytes;
                ok = pf_wait(bar_acc_empty + 8 * acc, pha ^ 1u, give_up, limit);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    ok = ok && pf_wait(bar_full + 8 * (2 * pair + half), ph, give_up, limit);
                    if (!ok)
                        break;
                    tc_fence_after();
                    const uint32_t t = ta + (uint32_t)half * kStageBytes;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_i8(d, smem_desc_sw128(t + (uint32_t)kk * 32u), smem_desc_sw128(t + kABytes + (uint32_t)kk * 32u), C::kIdesc,
                                (half | kk) ? 1u : 0u);
                    umma_commit(bar_empty + 8 * (2 * pair + half));  // the stage may be refilled when these have read it
                }
                if (ok)
                    umma_commit(bar_acc_full + 8 * acc);             // the group's sums are complete
                pair += 2;
                if (pair >= C::kPairs) {
                    pair -= C::kPairs;
                    ph ^= 1u;
                }
                acc += 2;
                if (acc >= kAccs) {
                    acc -= kAccs;
                    pha ^= 1u;
                }
            }
            if (!ok || *give_up) {
                umma_commit(bar_fin + 8 * b);
                const long long c0 = sm_clock();
                while (!mbar_try_wait(bar_fin + 8 * b, 0) && sm_clock() - c0 < limit) {
                }
            }
        }
    } else if (warp >= 4) {
        // ---- epilogue: thread = one row of the tile and half of the tokens, their sums in registers
        constexpr int kTH = C::kHalf, kCh = C::kChunk;
        // The table of units is the epilogue's alone: its loads (two trips to the L2) run beside the first tiles' copies and products.
        const int et = tid - 128;
        if (et < TT) {
            // RootMeanSquare.java:25-35: the scalar of the RMSNorm in front multiplies every unit of the token
            float ss = 1.0f;
            if (p.ssq != nullptr) {
                float tot = 0.f;
                for (int y = 0; y < p.nssq; ++y)
                    tot += p.ssq[(tb * p.nssq + y) * kT + et];
                tot = __fdiv_rn(tot, (float)p.n);
                tot = __fadd_rn(tot, 1e-5f);
                ss = __fdiv_rn(1.0f, __fsqrt_rn(tot));
            }
            s_ss[et] = ss;
        }
        named_barrier_sync(1, 32 * kEpiWarps);
        for (int i = et; i < G * TT; i += 32 * kEpiWarps) {
            const int g = i / TT, t = i - g * TT;
            const float2 u = p.ux[(size_t)(tb * G + g) * kT + t];
            s_ux[i] = make_float2(u.x * s_ss[t], u.y);
        }
        named_barrier_sync(1, 32 * kEpiWarps);
        const int q = warp & 3;                               // the quarter of tensor memory this warp may read
        const int th = (warp - 4) >> 2;                       // which half of the tokens
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(th * kTH);
        typename C::Count it = 0;
        bool ok = true;
        for (int tile = first; tile < ntiles && ok; tile += stride) {
            int sg = 0, m0 = (tile / p.ksplit) * kTileM;
            while (m0 >= p.seg[sg].rows) {
                m0 -= p.seg[sg].rows;
                ++sg;
            }
            const int z = tile % p.ksplit, g0 = z * gper, g1 = min(G, g0 + gper);
            const int row = m0 + q * 32 + lane;
            const float2 *hrow = p.seg[sg].hdr + (size_t)row * G;
            float acc[kTH];
#pragma unroll
            for (int t = 0; t < kTH; ++t)
                acc[t] = 0.f;
            // The (min, scale) pairs of the row come from HBM, 8 bytes per group and row: they are asked for four
            // groups ahead, or every group would wait one memory latency for its own pair.
            const int glast = g1 > g0 ? g1 - 1 : 0;
            float2 msq[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                msq[j] = hrow[min(g0 + j, glast)];
            for (int gb = g0; gb < g1 && ok; gb += 4) {
                float2 nxt[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    nxt[j] = hrow[min(gb + 4 + j, glast)];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int g = gb + j;
                    if (g >= g1 || !ok)
                        continue;
                    const float2 ms = msq[j];
                    const int b = (int)(it % kAccs);
                    const uint32_t pha = (uint32_t)((it / kAccs) & 1);
                    // one answer for the warp: the loads below are the whole warp's
                    if (!__all_sync(0xffffffffu, pf_wait(bar_acc_full + 8 * b, pha, give_up, limit))) {
                        ok = false;
                        continue;
                    }
                    tc_fence_after();
                    const uint32_t tacc = trow + (uint32_t)(b * C::kAccDist);
                    const float2 *ux = s_ux + g * TT + th * kTH;
                    // in parts: registers
#pragma unroll
                    for (int c = 0; c < kTH; c += kCh) {
                        uint32_t s0[kCh], s1[kCh], s2[kCh];
                        if constexpr (kCh == 16) {
                            tmem_ld16(tacc + c, s0);
                            tmem_ld16(tacc + TT + c, s1);
                            tmem_ld16(tacc + 2 * TT + c, s2);
                        } else {
                            tmem_ld8(tacc + c, s0);
                            tmem_ld8(tacc + TT + c, s1);
                            tmem_ld8(tacc + 2 * TT + c, s2);
                        }
                        tmem_ld_wait();
                        if (c + kCh == kTH) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0)
                                mbar_arrive(bar_acc_empty + 8 * b);
                        }
#pragma unroll
                        for (int k = 0; k < kCh; ++k) {
                            // |s0|, |s1| <= 256 * 255 * 128: the two lower limbs together still fit 32 bits
                            const float low = (float)((int)s1[k] * 256 + (int)s0[k]);
                            const float dsum = fmaf((float)(int)s2[k], 65536.0f, low);
                            const float2 u = ux[c + k];
                            acc[c + k] += fmaf(ms.y, dsum, ms.x * u.y) * u.x;
                        }
                    }
                    ++it;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    msq[j] = nxt[j];
            }
            if (ok) {
                const int t0 = tb * kT + th * kTH;
                float *o = p.out + ((size_t)z * kT * p.tblocks + t0) * p.ldc + p.seg[sg].col0 + row;
#pragma unroll
                for (int t = 0; t < kTH; ++t)
                    if (t0 + t < p.nvalid)
                        o[(size_t)t * p.ldc] = acc[t];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1)
        tmem_dealloc(tmem, kTmemCols);
    if (tid == 0 && s_give_up)
        atomicOr(p.status, PF_DS_WAIT_TIMEOUT);
}

// ---------------------------------------------------------------------------------------------------------------
// activations -> limbs
// ---------------------------------------------------------------------------------------------------------------

enum { PF_IN_NORM = 0, PF_IN_ATTN = 1, PF_IN_SWIGLU = 2 };

struct PfLimbParams {
    float *a;              // [tokens][lda]: x (NORM, updated with the parts), h1 (SWIGLU); ATTN: unused
    const float *b;        // NORM: RMSNorm weights [n]; SWIGLU: h3 [tokens][lda]
    const float *parts;    // NORM: [nparts][tokens][lda] partial row sums of the matrix in front, added to x in this order;
                           // ATTN: [nparts][tokens][heads][head + 2] partial attention outputs (o, m, l) of the key ranges
    int nparts;
    int head;              // ATTN: head size
    int lda;
    int n;                 // elements per token (multiple of 256)
    int nvalid;
    int tpad;              // tokens of the chunk, whole blocks of 64 (distance of the parts)
    int tt;                // tokens of a block of the B operand: 64, or what the matrix kernel of a call of few tokens takes
    int8_t *limbs;         // [token block][3 * tt][n]
    float2 *ux;            // [token block][n / 256][64]: (value of one fixed-point unit, sum of the fixed-point activations)
    float *ssq;            // NORM: [token block][gridDim.y][64] partial sums of squares of the rows
};

constexpr int kLimbWarps = 4, kLimbThreads = 32 * kLimbWarps;

template <int MODE>
__global__ void __launch_bounds__(kLimbThreads) pf_limbs_kernel(const PfLimbParams p)
{
    // one quantisation group per warp, kLimbWarps groups per block: nothing loops, every load of the block is in
    // flight at once
    __shared__ float s_ssq[kLimbWarps];
    const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tpad = p.tpad, tb = t / kT, tl = t % kT;
    const int G = p.n >> 8;
    const bool live = t < p.nvalid;
    float ssq = 0.f;
    const int gi = blockIdx.y * kLimbWarps + warp;
    pdl_launch_dependents();
    float4 wn[2];
    if (MODE == PF_IN_NORM && gi < G) {          // the weights do not depend on the kernel in front
#pragma unroll
        for (int h = 0; h < 2; ++h)
            wn[h] = *reinterpret_cast<const float4 *>(p.b + gi * 256 + h * 128 + lane * 4);
    }
    pdl_wait();
    if (gi < G) {
        float v[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int e = gi * 256 + h * 128 + lane * 4;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live && MODE != PF_IN_ATTN)
                x = *reinterpret_cast<const float4 *>(p.a + (size_t)t * p.lda + e);
            if (MODE == PF_IN_ATTN && live) {
                // the key ranges' partial results of this element's head, merged in a fixed order
                const int hd = e / p.head, d = e - hd * p.head, heads = p.n / p.head, rec = p.head + 2;
                float mx = -FLT_MAX;
                for (int z = 0; z < p.nparts; ++z)
                    mx = fmaxf(mx, p.parts[((size_t)(z * tpad + t) * heads + hd) * rec + p.head]);
                float lsum = 0.f;
                for (int z = 0; z < p.nparts; ++z) {
                    const float *r = p.parts + ((size_t)(z * tpad + t) * heads + hd) * rec;
                    const float w = expf(r[p.head] - mx);
                    lsum = fmaf(w, r[p.head + 1], lsum);
                    x.x = fmaf(w, r[d], x.x); x.y = fmaf(w, r[d + 1], x.y); x.z = fmaf(w, r[d + 2], x.z); x.w = fmaf(w, r[d + 3], x.w);
                }
                x.x = __fdiv_rn(x.x, lsum); x.y = __fdiv_rn(x.y, lsum); x.z = __fdiv_rn(x.z, lsum); x.w = __fdiv_rn(x.w, lsum);
            }
            if (MODE == PF_IN_NORM && live && p.nparts > 0) {
                for (int z = 0; z < p.nparts; ++z) {
                    const float4 d4 = *reinterpret_cast<const float4 *>(p.parts + ((size_t)z * tpad + t) * p.lda + e);
                    x.x = __fadd_rn(x.x, d4.x); x.y = __fadd_rn(x.y, d4.y); x.z = __fadd_rn(x.z, d4.z); x.w = __fadd_rn(x.w, d4.w);
                }
                *reinterpret_cast<float4 *>(p.a + (size_t)t * p.lda + e) = x;   // the residual stream after the matrix in front
            }
            if (MODE == PF_IN_NORM) {
                const float4 w = wn[h];
                ssq = fmaf(x.x, x.x, ssq); ssq = fmaf(x.y, x.y, ssq); ssq = fmaf(x.z, x.z, ssq); ssq = fmaf(x.w, x.w, ssq);
                x.x = __fmul_rn(w.x, x.x); x.y = __fmul_rn(w.y, x.y); x.z = __fmul_rn(w.z, x.z); x.w = __fmul_rn(w.w, x.w);
            } else if (MODE == PF_IN_SWIGLU) {
                float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
                if (live)
                    y = *reinterpret_cast<const float4 *>(p.b + (size_t)t * p.lda + e);
                for (int z = 1; z < p.nparts && live; ++z) {   // split-K parts of h1 and h3, in order
                    const float4 xz = *reinterpret_cast<const float4 *>(p.a + ((size_t)z * tpad + t) * p.lda + e);
                    const float4 yz = *reinterpret_cast<const float4 *>(p.b + ((size_t)z * tpad + t) * p.lda + e);
                    x.x = __fadd_rn(x.x, xz.x); x.y = __fadd_rn(x.y, xz.y); x.z = __fadd_rn(x.z, xz.z); x.w = __fadd_rn(x.w, xz.w);
                    y.x = __fadd_rn(y.x, yz.x); y.y = __fadd_rn(y.y, yz.y); y.z = __fadd_rn(y.z, yz.z); y.w = __fadd_rn(y.w, yz.w);
                }
                // Silu.java:122-132 order: (value * sigmoid) * hb2
                x.x = __fmul_rn(__fmul_rn(x.x, sigmoid_accurate(x.x)), y.x);
                x.y = __fmul_rn(__fmul_rn(x.y, sigmoid_accurate(x.y)), y.y);
                x.z = __fmul_rn(__fmul_rn(x.z, sigmoid_accurate(x.z)), y.z);
                x.w = __fmul_rn(__fmul_rn(x.w, sigmoid_accurate(x.w)), y.w);
            }
            v[4 * h] = x.x; v[4 * h + 1] = x.y; v[4 * h + 2] = x.z; v[4 * h + 3] = x.w;
        }
        float amax = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            amax = fmaxf(amax, fabsf(v[q]));
        amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
        // 24-bit fixed point: one power-of-two scale per group, |x * f| <= 2^22 (the decode kernels' rule)
        int ex = (int)((__float_as_uint(amax) >> 23) & 0xffu) - 126;
        if (!(amax > 0.f) || !(amax < 3.0e38f))
            ex = 0;
        ex = max(-90, min(126, ex));
        const float f = __int_as_float((127 + 22 - ex) << 23);
        uint32_t z[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
            z[q] = ((uint32_t)__float2int_rn(v[q] * f) + 0x00008080u) ^ 0x00008080u;
        int s0 = 0, s1 = 0, s2 = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t t0 = __byte_perm(z[4 * h], z[4 * h + 1], 0x5140);
            const uint32_t t2 = __byte_perm(z[4 * h + 2], z[4 * h + 3], 0x5140);
            const uint32_t t1 = __byte_perm(z[4 * h], z[4 * h + 1], 0x0062);
            const uint32_t t3 = __byte_perm(z[4 * h + 2], z[4 * h + 3], 0x0062);
            const uint32_t l0 = __byte_perm(t0, t2, 0x5410), l1 = __byte_perm(t0, t2, 0x7632), l2 = __byte_perm(t1, t3, 0x5410);
            const size_t e = (size_t)gi * 256 + h * 128 + lane * 4;
            *reinterpret_cast<uint32_t *>(p.limbs + (size_t)((3 * tb + 0) * p.tt + tl) * p.n + e) = l0;
            *reinterpret_cast<uint32_t *>(p.limbs + (size_t)((3 * tb + 1) * p.tt + tl) * p.n + e) = l1;
            *reinterpret_cast<uint32_t *>(p.limbs + (size_t)((3 * tb + 2) * p.tt + tl) * p.n + e) = l2;
            s0 = dp4a_ones(l0, s0);
            s1 = dp4a_ones(l1, s1);
            s2 = dp4a_ones(l2, s2);
        }
        s0 = __reduce_add_sync(0xffffffffu, s0);
        s1 = __reduce_add_sync(0xffffffffu, s1);
        s2 = __reduce_add_sync(0xffffffffu, s2);
        if (lane == 0) {
            const float inv = __int_as_float((127 + ex - 22) << 23);   // value of one fixed-point unit
            const float xs = fmaf((float)s2, 65536.0f, fmaf((float)s1, 256.0f, (float)s0));
            p.ux[((size_t)tb * G + gi) * kT + tl] = live ? make_float2(inv, xs) : make_float2(0.f, 0.f);
        }
    }
    if (MODE == PF_IN_NORM) {
        // the row's sum of squares: per block here, summed in block order by the matrix kernel that needs it
        ssq = warp_sum(ssq);
        if (lane == 0)
            s_ssq[warp] = ssq;
        __syncthreads();
        if (tid == 0) {
            float tot = 0.f;
            for (int w = 0; w < kLimbWarps; ++w)
                tot += s_ssq[w];
            p.ssq[((size_t)tb * gridDim.y + blockIdx.y) * kT + tl] = tot;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// embedding rows, RoPE + cache rows
// ---------------------------------------------------------------------------------------------------------------

__global__ void pf_embed_kernel(const int *tokens, int nvalid, const float *emb, int dim, int vocab, float *x)
{
    const int t = blockIdx.x;
    pdl_launch_dependents();
    int tok = t < nvalid ? tokens[t] : 0;
    tok = min(max(tok, 0), vocab - 1);
    const float4 *src = reinterpret_cast<const float4 *>(emb + (size_t)tok * dim);
    float4 *dst = reinterpret_cast<float4 *>(x + (size_t)t * dim);
    for (int i = threadIdx.x; i < dim / 4; i += blockDim.x)
        dst[i] = t < nvalid ? src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
}

struct PfRopeParams {
    const float *qkv;      // [tokens][dim + 2 kv_dim]
    float *q;              // [tokens][dim]
    float *k_cache, *v_cache;   // layer base, [kv_head][seq][head]
    const float *rope_cos, *rope_sin;   // [seq][head / 2]
    int dim, kv_dim, head, seq_len, pos0, nvalid;
    int nparts;                         // split-K parts of qkv ([nparts][tokens][dim + 2 kv_dim]), summed here in order
    const int *pos_of, *seq_of;         // concurrent sequences: position and sequence of every token (else pos0 + t, one cache)
    long long seq_stride;               // floats between the caches of two sequences
};

__global__ void pf_rope_kv_kernel(PfRopeParams p)
{
    const int t = blockIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (t >= p.nvalid)
        return;
    const int pos = p.pos_of ? p.pos_of[t] : p.pos0 + t, half = p.head >> 1;
    if (p.seq_of) {
        p.k_cache += (size_t)p.seq_of[t] * p.seq_stride;
        p.v_cache += (size_t)p.seq_of[t] * p.seq_stride;
    }
    const float *row = p.qkv + (size_t)t * (p.dim + 2 * p.kv_dim);
    const float *cs = p.rope_cos + (size_t)pos * half, *sn = p.rope_sin + (size_t)pos * half;
    const int i = blockIdx.y * blockDim.x + threadIdx.x;      // one pair per thread
    if (i < (p.dim + 2 * p.kv_dim) / 2) {
        const int e = 2 * i;
        float v0 = row[e], v1 = row[e + 1];
        for (int z = 1; z < p.nparts; ++z) {
            const float *rz = row + (size_t)z * gridDim.x * (p.dim + 2 * p.kv_dim);
            v0 = __fadd_rn(v0, rz[e]);
            v1 = __fadd_rn(v1, rz[e + 1]);
        }
        if (e < p.dim + p.kv_dim) {
            const int r = e < p.dim ? e : e - p.dim;
            const int d = r % p.head;
            const float c = cs[d >> 1], s = sn[d >> 1];
            const float r0 = __fsub_rn(__fmul_rn(v0, c), __fmul_rn(v1, s));   // ApplyRope.java:61-92
            const float r1 = __fadd_rn(__fmul_rn(v0, s), __fmul_rn(v1, c));
            if (e < p.dim) {
                p.q[(size_t)t * p.dim + r] = r0;
                p.q[(size_t)t * p.dim + r + 1] = r1;
            } else {
                float *dst = p.k_cache + ((size_t)(r / p.head) * p.seq_len + pos) * p.head + d;
                dst[0] = r0;
                dst[1] = r1;
            }
        } else {
            const int r = e - p.dim - p.kv_dim;
            float *dst = p.v_cache + ((size_t)(r / p.head) * p.seq_len + pos) * p.head + (r % p.head);
            dst[0] = v0;
            dst[1] = v1;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// causal attention of the chunk's queries
// ---------------------------------------------------------------------------------------------------------------

struct PfAttnParams {
    const float *q;        // [tokens][dim] after RoPE
    const float *k_cache, *v_cache;
    float *parts;          // [nsplit][tpad][heads][head + 2]: unnormalised output, running maximum, sum of the key range
    int dim, kv_mul, seq_len, pos0, nvalid, nsplit;
    int tpad;              // tokens of the chunk, whole blocks of 64
    int timeout_us;
    unsigned int *status;
};

// Block = (head, 128 queries, one range of key tiles), on the tensor cores without giving up FP32: every operand is
// the sum of three bf16 numbers of 8 significant bits (24 in all, exact), and the six products of pieces that reach
// 2^-24 of the result are added, the smallest first, into a fresh FP32 accumulator per tile; the running output is
// kept and rescaled in FP32 registers, so no sum is longer than one tile in the tensor cores' accumulator.
//
//   warps 0-3    softmax, one warp per scheduler: thread = query row; S from tensor memory, online maximum and sum, the three
//                pieces of P back into tensor memory (the A operand of the second product).  1 / sqrt(head size) is applied
//                to Q, and only tiles that need masks have them
//   warps 4-11   K and V of the tile from global memory through registers into their pieces in shared memory (V
//                transposed: both operands K-major, 128-byte swizzle); the output row of the query in registers
//   warp 12      issue, the longest of the roles: S(j + 1) = Q K' while the softmax works on tile j, then O(j) = P V
//
// Six bf16 products of 128 x 64 x HEAD, twice per tile, are 3072 tensor-core cycles at head size 128; on the FP32 units
// the same tile takes 16384 cycles at best.  A tile takes 8000, 6900 of them the issue of its 72 instructions (48 wider
// ones took as long); the softmax warps wait for 3400 of theirs.  3840 tokens through 16 layers of the 7B shape: 144 ms with
// the FP32 kernel before this one (4 x 4 scores per thread), 88 ms with it; scale and masks as above: 83.7 -> 81.8 ms.
// Error against float64 the same or lower (3.4e-6 against 3.6e-6 of a row of V behind it, mean over head sizes 64 and 128
// and peaked softmaxes).
constexpr int kAttnQ = 128;      // queries per block: the rows of one accumulator
constexpr int kAttnKeys = 64;    // keys per tile
constexpr int kAttnSoft = 4, kAttnCvt = 8;              // warps by role
constexpr int kAttnThreads = 32 * (kAttnSoft + kAttnCvt + 1);
constexpr int kAttnColO = 128, kAttnColP = 256;         // tensor memory: S 2 x 64 columns, O, P 3 x 32 columns

template <int HEAD>
constexpr size_t attn_smem_bytes()
{
    return (size_t)3 * (kAttnQ + 2 * kAttnKeys) * HEAD * 2 + 1024;      // pieces of Q, K and V, alignment
}

// c f32, a and b bf16, both K-major, M 128
__host__ __device__ constexpr uint32_t attn_idesc(int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kAttnQ >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// A from tensor memory: two consecutive K elements per 32-bit column
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t *r)
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::"r"(r[0]),
        "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_st_wait()
{
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// A pair of floats as three pairs of bf16 that add up to them: each difference is exact, and what the third piece has to
// hold fits its 8 bits.  The first two pieces saturate: a float above the largest bf16 is then the sum of finite pieces,
// and of an infinite one only the third piece is infinite, which meets nothing but the other operand's first piece, so that
// the product is the infinity of the right sign and not infinity - infinity.
__device__ __forceinline__ void split_bf16(float a, float b, uint32_t (&piece)[3])
{
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (i < 2)
            asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(piece[i]) : "f"(b), "f"(a));
        else
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(piece[i]) : "f"(b), "f"(a));
        a -= __uint_as_float(piece[i] << 16);
        b -= __uint_as_float(piece[i] & 0xffff0000u);
    }
}

// Eight floats to the 16-byte chunk `chunk` of row `row` of a swizzled K-major tile, one tile per piece.
__device__ __forceinline__ void store_pieces(unsigned char *tile, uint32_t piece_bytes, int row, int chunk, const float *v)
{
    uint32_t w[4][3];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        split_bf16(v[2 * i], v[2 * i + 1], w[i]);
    unsigned char *dst = tile + row * 128 + ((chunk ^ (row & 7)) << 4);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        *reinterpret_cast<uint4 *>(dst + i * piece_bytes) = make_uint4(w[0][i], w[1][i], w[2][i], w[3][i]);
}

// The pairs of pieces whose product is added, the smallest first (0: the leading eight bits).
__device__ __constant__ const int kPairA[6] = {2, 1, 0, 1, 0, 0}, kPairB[6] = {0, 1, 2, 0, 1, 0};

template <int HEAD>
__global__ void __launch_bounds__(kAttnThreads, 1) pf_attention_kernel(const PfAttnParams p)
{
    constexpr int HB = HEAD / 64;                            // 64-column blocks of a row of Q and K
    constexpr uint32_t kQBlock = kAttnQ * 128, kKBlock = kAttnKeys * 128, kVPiece = HEAD * 128;
    constexpr uint32_t kQPiece = HB * kQBlock, kKPiece = HB * kKBlock;
    constexpr int NU = HEAD / 32;                            // units of eight elements per converting thread and tile
    constexpr int NO = HEAD / 2;                             // output elements per converting thread
    extern __shared__ unsigned char pf_att_smem[];
    __shared__ __align__(8) unsigned long long s_bar[11];
    __shared__ uint32_t s_tmem;
    __shared__ int s_give_up;
    __shared__ float s_alpha[2][kAttnQ];

    const int h = blockIdx.x, q0 = blockIdx.y * kAttnQ, z = blockIdx.z;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (q0 >= p.nvalid)
        return;
    const uint32_t base = (smem_u32(pf_att_smem) + 1023u) & ~1023u;
    unsigned char *gen = pf_att_smem + (base - smem_u32(pf_att_smem));
    unsigned char *gQ = gen, *gK = gQ + 3 * kQPiece, *gV = gK + 3 * kKPiece;
    const uint32_t aQ = base, aK = aQ + 3 * kQPiece, aV = aK + 3 * kKPiece;
    const uint32_t bar = smem_u32(&s_bar[0]);
    const uint32_t b_k = bar, b_v = bar + 8, b_p = bar + 16, b_pv = bar + 24, b_qk = bar + 32, b_s = bar + 48, b_a = bar + 64,
                   b_fin = bar + 80;                         // b_qk, b_s, b_a: two each, by the tile's parity
    const long long limit = 2000ll * (long long)p.timeout_us;
    volatile int *give_up = &s_give_up;

    const int kvh = h / p.kv_mul;
    const float *kbase = p.k_cache + (size_t)kvh * p.seq_len * HEAD;
    const float *vbase = p.v_cache + (size_t)kvh * p.seq_len * HEAD;
    const int nkeys = p.pos0 + min(q0 + kAttnQ, p.nvalid);  // keys 0 .. position of the block's last query
    const int tiles = (nkeys + kAttnKeys - 1) / kAttnKeys;
    const int tper = (tiles + p.nsplit - 1) / p.nsplit;
    const int t_lo = z * tper, n = max(0, min(tiles, t_lo + tper) - t_lo);

    if (tid == 0) {
        mbar_init(b_k, kAttnCvt);
        mbar_init(b_v, kAttnCvt);
        mbar_init(b_p, kAttnSoft);
        mbar_init(b_pv, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(b_qk + 8 * i, 1);
            mbar_init(b_s + 8 * i, kAttnSoft);
            mbar_init(b_a + 8 * i, kAttnSoft);
        }
        mbar_init(b_fin, 1);
        mbar_fence_init();
        s_give_up = 0;
    }
    pdl_launch_dependents();
    pdl_wait();
    if (warp == kAttnSoft + kAttnCvt) {
        tmem_alloc(smem_u32(&s_tmem), kTmemCols);
        tmem_relinquish();
    }
    const float root = sqrtf((float)HEAD);
    for (int u = tid; u < kAttnQ * HEAD / 8; u += kAttnThreads) {
        const int r = u / (HEAD / 8), c8 = u % (HEAD / 8);
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (q0 + r < p.nvalid) {
            const float4 *src = reinterpret_cast<const float4 *>(p.q + (size_t)(q0 + r) * p.dim + h * HEAD + c8 * 8);
            const float4 x = src[0], y = src[1];
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
            // AttentionLoop: score / sqrt(head_size); on the query, once per element instead of once per score
#pragma unroll
            for (int i = 0; i < 8; ++i)
                v[i] = __fdiv_rn(v[i], root);
        }
        store_pieces(gQ + (c8 >> 3) * kQBlock, kQPiece, r, c8 & 7, v);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int heads = p.dim / HEAD;

    if (warp < kAttnSoft) {
        // ---- softmax: thread = query row
        const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
        const int row = warp * 32 + lane, qpos = p.pos0 + q0 + row;
        float m = -FLT_MAX, l = 0.f;
        for (int j = 0; j < n; ++j) {
            const int k0 = (t_lo + j) * kAttnKeys;
            if (!__all_sync(0xffffffffu, pf_wait(b_qk + 8 * (j & 1), (uint32_t)((j >> 1) & 1), give_up, limit)))
                break;
            tc_fence_after();
            uint32_t raw[64];
#pragma unroll
            for (int c = 0; c < 4; ++c)
                tmem_ld16(trow + (uint32_t)((j & 1) * kAttnKeys + 16 * c), raw + 16 * c);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(b_s + 8 * (j & 1));
            const int last = qpos - k0;                      // keys past it are masked
            if (!__all_sync(0xffffffffu, last >= kAttnKeys - 1)) {
#pragma unroll
                for (int c = 0; c < 64; ++c)
                    raw[c] = c <= last ? raw[c] : __float_as_uint(-FLT_MAX);
            }
            float mx4[4] = {-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
#pragma unroll
            for (int c = 0; c < 64; ++c)
                mx4[c & 3] = fmaxf(mx4[c & 3], __uint_as_float(raw[c]));
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            const float mn = fmaxf(m, mx);
            const float alpha = expf(m - mn);
            const float shift = mn > -FLT_MAX ? mn : 0.f;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 64; ++c) {
                // (masked: zero, also where a row has no key in this range yet and mn is -FLT_MAX itself)
                const float pv = expf(__uint_as_float(raw[c]) - shift);
                raw[c] = __float_as_uint(pv);
                sum[c & 3] += pv;
            }
            l = l * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
            m = mn;
            if (j > 0 && !__all_sync(0xffffffffu, pf_wait(b_pv, (uint32_t)((j - 1) & 1), give_up, limit)))
                break;
            tc_fence_after();
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t w[3][16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    uint32_t pc[3];
                    split_bf16(__uint_as_float(raw[32 * half + 2 * i]), __uint_as_float(raw[32 * half + 2 * i + 1]), pc);
                    w[0][i] = pc[0]; w[1][i] = pc[1]; w[2][i] = pc[2];
                }
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    tmem_st16(trow + (uint32_t)(kAttnColP + 32 * i + 16 * half), w[i]);
            }
            tmem_st_wait();
            s_alpha[j & 1][row] = alpha;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(b_p);
                mbar_arrive(b_a + 8 * (j & 1));
            }
        }
        if (q0 + row < p.nvalid && !*give_up) {
            float *rec = p.parts + ((size_t)(z * p.tpad + q0 + row) * heads + h) * (HEAD + 2);
            rec[HEAD] = m;
            rec[HEAD + 1] = l;
        }
    } else if (warp < kAttnSoft + kAttnCvt) {
        // ---- operands and output: K and V unit by unit, output row q, half of its elements
        const int ct = tid - 32 * kAttnSoft, quarter = warp & 3, part = (warp - kAttnSoft) >> 2;
        const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(kAttnColO + part * NO);
        const int row = quarter * 32 + lane;
        float o[NO];
#pragma unroll
        for (int i = 0; i < NO; ++i)
            o[i] = 0.f;
        float x[NU][8];
        auto load_k = [&](int j) {
            const int k0 = (t_lo + j) * kAttnKeys;
#pragma unroll
            for (int i = 0; i < NU; ++i) {
                const int u = ct + 256 * i, key = u / (HEAD / 8), c8 = u % (HEAD / 8);
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
                if (k0 + key < nkeys) {
                    const float4 *src = reinterpret_cast<const float4 *>(kbase + (size_t)(k0 + key) * HEAD + c8 * 8);
                    a = src[0];
                    b = src[1];
                }
                x[i][0] = a.x; x[i][1] = a.y; x[i][2] = a.z; x[i][3] = a.w; x[i][4] = b.x; x[i][5] = b.y; x[i][6] = b.z; x[i][7] = b.w;
            }
        };
        auto load_v = [&](int j) {
            const int k0 = (t_lo + j) * kAttnKeys;
#pragma unroll
            for (int i = 0; i < NU; ++i) {
                const int u = ct + 256 * i, d = u % HEAD, key = 8 * (u / HEAD);
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    x[i][e] = k0 + key + e < nkeys ? vbase[(size_t)(k0 + key + e) * HEAD + d] : 0.f;
            }
        };
        auto publish = [&](uint32_t b) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                mbar_arrive(b);
        };
        auto store_k = [&]() {
#pragma unroll
            for (int i = 0; i < NU; ++i) {
                const int u = ct + 256 * i, key = u / (HEAD / 8), c8 = u % (HEAD / 8);
                store_pieces(gK + (c8 >> 3) * kKBlock, kKPiece, key, c8 & 7, x[i]);
            }
            publish(b_k);
        };
        auto add_output = [&](int j) -> bool {               // O(j) of the tensor cores into the running output
            if (!__all_sync(0xffffffffu, pf_wait(b_a + 8 * (j & 1), (uint32_t)((j >> 1) & 1), give_up, limit)) ||
                !__all_sync(0xffffffffu, pf_wait(b_pv, (uint32_t)(j & 1), give_up, limit)))
                return false;
            tc_fence_after();
            const float alpha = s_alpha[j & 1][row];
#pragma unroll
            for (int c = 0; c < NO; c += 16) {
                uint32_t t[16];
                tmem_ld16(trow + (uint32_t)c, t);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    o[c + i] = fmaf(o[c + i], alpha, __uint_as_float(t[i]));
            }
            tc_fence_before();
            return true;
        };
        if (n > 0) {
            load_k(0);
            store_k();
        }
        if (n > 1)
            load_k(1);
        bool ok = true;
        for (int j = 0; j < n; ++j) {
            if (j + 1 < n) {
                ok = __all_sync(0xffffffffu, pf_wait(b_qk + 8 * (j & 1), (uint32_t)((j >> 1) & 1), give_up, limit));
                if (!ok)
                    break;
                store_k();
            }
            load_v(j);
            if (j > 0) {
                ok = add_output(j - 1);
                if (!ok)
                    break;
            }
#pragma unroll
            for (int i = 0; i < NU; ++i) {
                const int u = ct + 256 * i;
                store_pieces(gV, kVPiece, u % HEAD, u / HEAD, x[i]);
            }
            publish(b_v);
            if (j + 2 < n)
                load_k(j + 2);
        }
        if (ok && n > 0)
            ok = add_output(n - 1);
        if (ok && q0 + row < p.nvalid) {
            float *rec = p.parts + ((size_t)(z * p.tpad + q0 + row) * heads + h) * (HEAD + 2) + part * NO;
#pragma unroll
            for (int i = 0; i < NO; i += 2)                  // records are 8-byte aligned (HEAD + 2 floats each)
                *reinterpret_cast<float2 *>(rec + i) = make_float2(o[i], o[i + 1]);
        }
    } else if (lane == 0) {
        // ---- tensor-core issue: one lane
        bool ok = true;
        for (int j = 0; j <= n && n > 0; ++j) {
            if (j < n) {
                ok = pf_wait(b_k, (uint32_t)(j & 1), give_up, limit) &&
                     (j < 2 || pf_wait(b_s + 8 * (j & 1), (uint32_t)(((j >> 1) - 1) & 1), give_up, limit));
                if (!ok)
                    break;
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)((j & 1) * kAttnKeys);
#pragma unroll 1
                for (int i = 0; i < 6; ++i) {
                    const uint32_t ta = aQ + (uint32_t)kPairA[i] * kQPiece, tb = aK + (uint32_t)kPairB[i] * kKPiece;
#pragma unroll
                    for (int kk = 0; kk < HEAD / 16; ++kk)
                        umma_bf16(d, smem_desc_sw128(ta + (kk >> 2) * kQBlock + (kk & 3) * 32u),
                                  smem_desc_sw128(tb + (kk >> 2) * kKBlock + (kk & 3) * 32u), attn_idesc(kAttnKeys), (i | kk) ? 1u : 0u);
                }
                umma_commit(b_qk + 8 * (j & 1));
            }
            if (j > 0) {
                ok = pf_wait(b_p, (uint32_t)((j - 1) & 1), give_up, limit) && pf_wait(b_v, (uint32_t)((j - 1) & 1), give_up, limit);
                if (!ok)
                    break;
                tc_fence_after();
#pragma unroll 1
                for (int i = 0; i < 6; ++i) {
                    const uint32_t ta = tmem + kAttnColP + 32u * (uint32_t)kPairA[i], tb = aV + (uint32_t)kPairB[i] * kVPiece;
#pragma unroll
                    for (int kk = 0; kk < kAttnKeys / 16; ++kk)
                        umma_bf16_ts(tmem + kAttnColO, ta + 8u * kk, smem_desc_sw128(tb + kk * 32u), attn_idesc(HEAD), (i | kk) ? 1u : 0u);
                }
                umma_commit(b_pv);
            }
        }
        if (!ok || *give_up) {
            umma_commit(b_fin);
            const long long c0 = sm_clock();
            while (!mbar_try_wait(b_fin, 0) && sm_clock() - c0 < limit) {
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kAttnSoft + kAttnCvt)
        tmem_dealloc(tmem, kTmemCols);
    if (tid == 0 && s_give_up)
        atomicOr(p.status, PF_DS_WAIT_TIMEOUT);
}

// ---------------------------------------------------------------------------------------------------------------
// concurrent sequences: one decode step of up to 64 (sequence, position) pairs on one sweep over the weights
// ---------------------------------------------------------------------------------------------------------------

struct BdAttnParams {
    const float *q;                     // [64][dim] after RoPE
    const float *k_cache, *v_cache;     // layer base of sequence 0, [kv_head][seq][head]
    long long seq_stride;
    const int *pos_of, *seq_of;
    float *parts;                       // [nsplit][64][heads][head + 2]: unnormalised output, maximum, sum of the key range
    int dim, kv_mul, seq_len, nvalid, nsplit;
};

constexpr int kBdWarps = 4, kBdThreads = 32 * kBdWarps;
constexpr int kBdKeys = 8;              // keys per warp and round: eight lanes share a key, four keys side by side, two deep

// Block = (head, token, one of nsplit key ranges): every token has its own cache and length.  Bound by the K and V bytes:
// a lane asks for all of its 16 (head 128) pieces of two keys' K and V rows before it needs the first, every row is read
// as whole 128-byte lines, and the online softmax runs per group of eight lanes, so that nothing but three shuffles per
// score crosses lanes until the end.  A step of 4 sequences of 600 to 1500 positions through 16 layers of the 7B shape:
// 5.78 ms with one block per (head, token) and a lane per key, 2.72 ms with this; 64 sequences of 10 to 200: 4.56 and 3.57.
template <int HEAD>
__global__ void __launch_bounds__(kBdThreads) bd_attention_kernel(const BdAttnParams p)
{
    constexpr int NV = HEAD / 32;       // float4 pieces of a row per lane
    __shared__ float s_m[kBdWarps], s_l[kBdWarps];
    __shared__ __align__(16) float s_o[kBdWarps][HEAD];
    const int h = blockIdx.x, t = blockIdx.y, z = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    pdl_wait();
    const int keys = p.pos_of[t] + 1;
    const int per = ((keys + p.nsplit - 1) / p.nsplit + kBdWarps * kBdKeys - 1) / (kBdWarps * kBdKeys) * (kBdWarps * kBdKeys);
    const int k_lo = z * per, k_hi = min(keys, k_lo + per);
    const size_t cache = (size_t)p.seq_of[t] * p.seq_stride + (size_t)(h / p.kv_mul) * p.seq_len * HEAD;
    const int sub = lane & 7, grp = lane >> 3;
    const float4 *kbase = reinterpret_cast<const float4 *>(p.k_cache + cache) + sub;
    const float4 *vbase = reinterpret_cast<const float4 *>(p.v_cache + cache) + sub;
    float4 q[NV], o[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        q[i] = reinterpret_cast<const float4 *>(p.q + (size_t)t * p.dim + h * HEAD)[sub + 8 * i];
        o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float root = sqrtf((float)HEAD);
    float m = -FLT_MAX, l = 0.f;
    for (int k0 = k_lo + warp * kBdKeys; k0 < k_hi; k0 += kBdWarps * kBdKeys) {
        float4 kv[2][NV], vv[2][NV];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const size_t key = (size_t)min(k0 + grp + 4 * u, k_hi - 1) * (HEAD / 4);
#pragma unroll
            for (int i = 0; i < NV; ++i)
                kv[u][i] = __ldcs(kbase + key + 8 * i);
#pragma unroll
            for (int i = 0; i < NV; ++i)
                vv[u][i] = __ldcs(vbase + key + 8 * i);
        }
        float sc[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            float a = 0.f, b = 0.f;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                a = fmaf(q[i].x, kv[u][i].x, a); b = fmaf(q[i].y, kv[u][i].y, b);
                a = fmaf(q[i].z, kv[u][i].z, a); b = fmaf(q[i].w, kv[u][i].w, b);
            }
            sc[u] = a + b;
#pragma unroll
            for (int x = 1; x < 8; x <<= 1)
                sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], x);
            sc[u] = k0 + grp + 4 * u < k_hi ? __fdiv_rn(sc[u], root) : -FLT_MAX;
        }
        const float mn = fmaxf(m, fmaxf(sc[0], sc[1]));
        const float alpha = expf(m - mn);
        const float w0 = sc[0] > -FLT_MAX ? expf(sc[0] - mn) : 0.f, w1 = sc[1] > -FLT_MAX ? expf(sc[1] - mn) : 0.f;
        l = l * alpha + (w0 + w1);
        m = mn;
        // a key past the range weighs nothing, whatever its row holds
        const bool in0 = w0 > 0.f, in1 = w1 > 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            o[i].x *= alpha; o[i].y *= alpha; o[i].z *= alpha; o[i].w *= alpha;
            if (in0) {
                o[i].x = fmaf(w0, vv[0][i].x, o[i].x); o[i].y = fmaf(w0, vv[0][i].y, o[i].y);
                o[i].z = fmaf(w0, vv[0][i].z, o[i].z); o[i].w = fmaf(w0, vv[0][i].w, o[i].w);
            }
            if (in1) {
                o[i].x = fmaf(w1, vv[1][i].x, o[i].x); o[i].y = fmaf(w1, vv[1][i].y, o[i].y);
                o[i].z = fmaf(w1, vv[1][i].z, o[i].z); o[i].w = fmaf(w1, vv[1][i].w, o[i].w);
            }
        }
    }
    // the warp's four groups, then the warps, each in a fixed order
    float mw = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
    mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, 16));
    const float scale = expf(m - mw);
    l *= scale;
    l += __shfl_xor_sync(0xffffffffu, l, 8);
    l += __shfl_xor_sync(0xffffffffu, l, 16);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        float e[4] = {o[i].x * scale, o[i].y * scale, o[i].z * scale, o[i].w * scale};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            e[c] += __shfl_xor_sync(0xffffffffu, e[c], 8);
            e[c] += __shfl_xor_sync(0xffffffffu, e[c], 16);
        }
        if (grp == 0)
            *reinterpret_cast<float4 *>(&s_o[warp][4 * (sub + 8 * i)]) = make_float4(e[0], e[1], e[2], e[3]);
    }
    if (lane == 0) {
        s_m[warp] = mw;
        s_l[warp] = l;
    }
    __syncthreads();
    float mt = s_m[0];
#pragma unroll
    for (int w = 1; w < kBdWarps; ++w)
        mt = fmaxf(mt, s_m[w]);
    float *rec = p.parts + ((size_t)(z * kT + t) * (p.dim / HEAD) + h) * (HEAD + 2);
    if (tid < HEAD) {
        float acc = 0.f;
#pragma unroll
        for (int w = 0; w < kBdWarps; ++w)
            acc = fmaf(expf(s_m[w] - mt), s_o[w][tid], acc);
        rec[tid] = acc;
    }
    if (tid == 0) {
        float lt = 0.f;
#pragma unroll
        for (int w = 0; w < kBdWarps; ++w)
            lt = fmaf(expf(s_m[w] - mt), s_l[w], lt);
        rec[HEAD] = mt;
        rec[HEAD + 1] = lt;
    }
}

// Key ranges per (head, token): enough blocks for six on every SM.  The captured step serves all lengths, so the choice knows
// the number of entries only: ranges that a short sequence leaves empty cost a block that ends at once, and a long sequence
// among many short ones (from 28 entries at 32 heads on: one range) is scanned by one block per head.
int bd_splits(int heads, int nv, int sms)
{
    const int ns = (6 * sms) / (heads * nv);
    return ns < 1 ? 1 : (ns > kMaxParts ? kMaxParts : ns);
}

// x after the last layer (with the partial row sums of its W2), RMSNorm with the final weights
// (RootMeanSquare.java:25-35, WeightNormalizeAndScale.java:71-74), written as three bf16 pieces [3][64][dim]: the
// classifier's B operand.
__global__ void __launch_bounds__(256) bd_final_norm_kernel(float *x, const float *parts, int nparts, const float *w, int dim, int nvalid,
                                                            uint32_t *pieces)
{
    __shared__ float s_red[8];
    const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    pdl_wait();
    float ssq = 0.f;
    for (int i = tid; i < dim / 2; i += 256) {
        float2 v = make_float2(0.f, 0.f);
        if (t < nvalid)
            v = reinterpret_cast<const float2 *>(x + (size_t)t * dim)[i];
        for (int z = 0; z < nparts && t < nvalid; ++z) {
            const float2 d = reinterpret_cast<const float2 *>(parts + ((size_t)z * kT + t) * dim)[i];
            v.x = __fadd_rn(v.x, d.x);
            v.y = __fadd_rn(v.y, d.y);
        }
        reinterpret_cast<float2 *>(x + (size_t)t * dim)[i] = v;
        ssq = fmaf(v.x, v.x, ssq);
        ssq = fmaf(v.y, v.y, ssq);
    }
    ssq = warp_sum(ssq);
    if (lane == 0)
        s_red[warp] = ssq;
    __syncthreads();
    float tot = 0.f;
    for (int k = 0; k < 8; ++k)
        tot += s_red[k];
    tot = __fdiv_rn(tot, (float)dim);
    tot = __fadd_rn(tot, 1e-5f);
    const float ss = __fdiv_rn(1.0f, __fsqrt_rn(tot));
    for (int i = tid; i < dim / 2; i += 256) {
        const float2 v = reinterpret_cast<const float2 *>(x + (size_t)t * dim)[i], g = reinterpret_cast<const float2 *>(w)[i];
        uint32_t pc[3];
        split_bf16(__fmul_rn(g.x, __fmul_rn(ss, v.x)), __fmul_rn(g.y, __fmul_rn(ss, v.y)), pc);
#pragma unroll
        for (int k = 0; k < 3; ++k)
            pieces[((size_t)k * kT + t) * (dim / 2) + i] = pc[k];
    }
}

// logits[t][v] = sum_k wcls[v][k] * xn[t][k] for 64 tokens (the classifier is not quantised,
// TransformerWeights.java:25,41,122) on the tensor cores, FP32 operands in three bf16 pieces as in the attention above:
// per 64 columns of K, W's leading pieces times all three of x (N 192), the second times two (N 128), the third times one
// (N 64), into one accumulator per piece of x.  The accumulator starts anew every 64 columns and is added to the row sums
// in FP32 registers, so that no long sum runs in the tensor cores.  The floor is the 4 bytes per weight from HBM (80 us at
// 32000 x 4096; 167 us with cold caches: two tiles on two thirds of the SMs, one on the others); the FMA kernel before it was bound by its 16.8 GFLOP and made a step 0.29 to 0.38 ms longer.
//
//   warps 0-7    W from HBM through registers (two blocks of 64 columns ahead) into its pieces in shared memory
//   warps 8-15   row sums: thread = vocabulary row, half of the tokens
//   warp 16      tensor-core issue;  warp 17: copies of x's pieces (TMA)
constexpr int kClsRows = 128, kClsCols = 64, kClsStages = 3, kClsCvt = 8, kClsEpi = 8;
constexpr int kClsThreads = 32 * (kClsCvt + kClsEpi + 2);
constexpr int kClsAPiece = kClsRows * 128, kClsABytes = 3 * kClsAPiece, kClsBBytes = kN * 128, kClsStage = kClsABytes + kClsBBytes;

struct BdClsParams {
    const float *wcls;
    int vocab, dim, nvalid;
    float *logits;         // [64][vocab]
    int timeout_us;
    unsigned int *status;
};

__global__ void __launch_bounds__(kClsThreads, 1) bd_classifier_kernel(const __grid_constant__ CUtensorMap map_x, const BdClsParams p)
{
    extern __shared__ unsigned char cls_smem[];
    __shared__ __align__(8) unsigned long long s_bar[3 * kClsStages + 5];
    __shared__ uint32_t s_tmem;
    __shared__ int s_give_up;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(cls_smem) + 1023u) & ~1023u;
    unsigned char *gen = cls_smem + (base - smem_u32(cls_smem));
    const uint32_t b_full = smem_u32(&s_bar[0]), b_empty = smem_u32(&s_bar[kClsStages]), b_x = smem_u32(&s_bar[2 * kClsStages]),
                   b_acc = smem_u32(&s_bar[3 * kClsStages]), b_free = b_acc + 16, b_fin = b_acc + 32;
    const long long limit = 2000ll * (long long)p.timeout_us;
    volatile int *give_up = &s_give_up;
    const int tiles = (p.vocab + kClsRows - 1) / kClsRows, nk = p.dim / kClsCols;
    const int total = ((tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x) * nk;   // blocks of columns of all the tiles

    if (tid == 0) {
        for (int s = 0; s < kClsStages; ++s) {
            mbar_init(b_full + 8 * s, kClsCvt);
            mbar_init(b_x + 8 * s, 1);
            mbar_init(b_empty + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(b_acc + 8 * b, 1);
            mbar_init(b_free + 8 * b, kClsEpi);
        }
        mbar_init(b_fin, 1);
        mbar_fence_init();
        s_give_up = 0;
    }
    pdl_launch_dependents();
    __syncthreads();

    if (warp < kClsCvt) {
        // unit: eight columns of a row; a row's 64 columns are 256 contiguous bytes
        float4 x[2][4][2];
        auto load = [&](int it, float4 (&d)[4][2]) {
            const int tile = (int)blockIdx.x + it / nk * (int)gridDim.x, k0 = it % nk * kClsCols;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int u = tid + 256 * i, v = tile * kClsRows + (u >> 3);
                d[i][0] = d[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (v < p.vocab) {
                    const float4 *src = reinterpret_cast<const float4 *>(p.wcls + (size_t)v * p.dim + k0 + 8 * (u & 7));
                    d[i][0] = __ldcs(src);
                    d[i][1] = __ldcs(src + 1);
                }
            }
        };
        auto store = [&](int it, const float4 (&d)[4][2]) -> bool {
            const int s = it % kClsStages;
            if (it == kClsStages)
                pdl_wait();
            if (!__all_sync(0xffffffffu, pf_wait(b_empty + 8 * s, (uint32_t)((it / kClsStages) & 1) ^ 1u, give_up, limit)))
                return false;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int u = tid + 256 * i;
                const float v[8] = {d[i][0].x, d[i][0].y, d[i][0].z, d[i][0].w, d[i][1].x, d[i][1].y, d[i][1].z, d[i][1].w};
                store_pieces(gen + (size_t)s * kClsStage, kClsAPiece, u >> 3, u & 7, v);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                mbar_arrive(b_full + 8 * s);
            return true;
        };
        // The weights do not depend on the kernel in front: no wait for it before the ring is full.  The stage after that is
        // freed by the roles that do wait; the time limit of waiting for it must not run while the kernel in front still does.
        if (total > 0)
            load(0, x[0]);
        if (total > 1)
            load(1, x[1]);
        for (int it = 0; it < total; it += 2) {
            if (!store(it, x[0]))
                break;
            if (it + 2 < total)
                load(it + 2, x[0]);
            if (it + 1 < total) {
                if (!store(it + 1, x[1]))
                    break;
                if (it + 3 < total)
                    load(it + 3, x[1]);
            }
        }
        pdl_wait();                                          // (a ring that was never full)
    } else if (warp == kClsCvt + kClsEpi + 1) {
        pdl_wait();
        if (lane == 0) {
            int it = 0;
            for (; it < total; ++it) {
                const int s = it % kClsStages;
                if (!pf_wait(b_empty + 8 * s, (uint32_t)((it / kClsStages) & 1) ^ 1u, give_up, limit))
                    break;
                mbar_arrive_expect_tx(b_x + 8 * s, kClsBBytes);
                tma_load_2d(base + (uint32_t)(s * kClsStage + kClsABytes), &map_x, it % nk * 128, 0, b_x + 8 * s);
            }
            if (*give_up) {
                // copies that nobody consumed must land before the block's shared memory goes away
                for (int i = max(0, it - kClsStages); i < it; ++i) {
                    const long long c0 = sm_clock();
                    while (!mbar_try_wait(b_x + 8 * (i % kClsStages), (uint32_t)((i / kClsStages) & 1)) && sm_clock() - c0 < limit) {
                    }
                }
            }
        }
    } else if (warp == kClsCvt + kClsEpi) {
        pdl_wait();
        tmem_alloc(smem_u32(&s_tmem), kTmemCols);
        tmem_relinquish();
        tc_fence_before();
        named_barrier_sync(1, 32 * (kClsEpi + 1));
        tc_fence_after();
        const uint32_t tmem = s_tmem;
        if (lane == 0) {
            bool ok = true;
            for (int it = 0; it < total; ++it) {
                const int s = it % kClsStages, b = it & 1;
                ok = pf_wait(b_free + 8 * b, (uint32_t)((it >> 1) & 1) ^ 1u, give_up, limit) &&
                     pf_wait(b_full + 8 * s, (uint32_t)((it / kClsStages) & 1), give_up, limit) &&
                     pf_wait(b_x + 8 * s, (uint32_t)((it / kClsStages) & 1), give_up, limit);
                if (!ok)
                    break;
                tc_fence_after();
                const uint32_t ta = base + (uint32_t)(s * kClsStage), tb = ta + kClsABytes, d = tmem + (uint32_t)b * kAccCols;
                // columns 64 i .. 64 i + 63 of the accumulator belong to piece i of x; the first instruction starts all of them
#pragma unroll
                for (int kk = 0; kk < kClsCols / 16; ++kk)
                    umma_bf16(d, smem_desc_sw128(ta + kk * 32u), smem_desc_sw128(tb + kk * 32u), attn_idesc(kN), kk ? 1u : 0u);
#pragma unroll
                for (int kk = 0; kk < kClsCols / 16; ++kk) {
                    umma_bf16(d, smem_desc_sw128(ta + kClsAPiece + kk * 32u), smem_desc_sw128(tb + kk * 32u), attn_idesc(2 * kT), 1u);
                    umma_bf16(d, smem_desc_sw128(ta + 2 * kClsAPiece + kk * 32u), smem_desc_sw128(tb + kk * 32u), attn_idesc(kT), 1u);
                }
                umma_commit(b_empty + 8 * s);
                umma_commit(b_acc + 8 * b);
            }
            if (!ok || *give_up) {
                umma_commit(b_fin);
                const long long c0 = sm_clock();
                while (!mbar_try_wait(b_fin, 0) && sm_clock() - c0 < limit) {
                }
            }
        }
    } else {
        pdl_wait();
        named_barrier_sync(1, 32 * (kClsEpi + 1));
        tc_fence_after();
        const int quarter = warp & 3, th = (warp - kClsCvt) >> 2;
        constexpr int kTH = kT / 2;           // tokens per thread
        const uint32_t trow = s_tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(th * kTH);
        float acc[kTH];
#pragma unroll
        for (int t = 0; t < kTH; ++t)
            acc[t] = 0.f;
        for (int it = 0; it < total; ++it) {
            const int b = it & 1;
            if (!__all_sync(0xffffffffu, pf_wait(b_acc + 8 * b, (uint32_t)((it >> 1) & 1), give_up, limit)))
                break;
            tc_fence_after();
            const uint32_t tacc = trow + (uint32_t)b * kAccCols;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t s0[16], s1[16], s2[16];
                tmem_ld16(tacc + 16 * half, s0);
                tmem_ld16(tacc + kT + 16 * half, s1);
                tmem_ld16(tacc + 2 * kT + 16 * half, s2);
                tmem_ld_wait();
                if (half == 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(b_free + 8 * b);
                }
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    acc[16 * half + k] += __uint_as_float(s0[k]) + (__uint_as_float(s1[k]) + __uint_as_float(s2[k]));
            }
            if (it % nk == nk - 1) {
                const int v = ((int)blockIdx.x + it / nk * (int)gridDim.x) * kClsRows + quarter * 32 + lane;
                float *o = p.logits + (size_t)th * kTH * p.vocab + v;
#pragma unroll
                for (int t = 0; t < kTH; ++t) {
                    if (v < p.vocab && th * kTH + t < p.nvalid)
                        o[(size_t)t * p.vocab] = acc[t];
                    acc[t] = 0.f;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kClsCvt + kClsEpi)
        tmem_dealloc(s_tmem, kTmemCols);
    if (tid == 0 && s_give_up)
        atomicOr(p.status, PF_DS_WAIT_TIMEOUT);
}

// First maximum of every token's logits (Sampler.java:46-57).
__global__ void __launch_bounds__(256) bd_argmax_kernel(const float *logits, int vocab, int nvalid, int *out)
{
    __shared__ float s_v[8];
    __shared__ int s_i[8];
    const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_wait();
    float bv = -FLT_MAX;
    int bi = 0x7fffffff;
    for (int i = tid; i < vocab; i += 256) {
        const float v = logits[(size_t)t * vocab + i];
        if (v > bv) {
            bv = v;
            bi = i;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) {
            bv = ov;
            bi = oi;
        }
    }
    if (lane == 0) {
        s_v[warp] = bv;
        s_i[warp] = bi;
    }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < 8; ++w)
            if (s_v[w] > bv || (s_v[w] == bv && s_i[w] < bi)) {
                bv = s_v[w];
                bi = s_i[w];
            }
        out[t] = bi;
    }
}

// ---------------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------------

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn()
{
    static std::once_flag once;
    static EncodeTiledFn fn = nullptr;
    std::call_once(once, [] {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    });
    return fn;
}

// Byte matrix [rows][k] (row pitch k), tiles of box_rows x 128 bytes, 128-byte swizzled in shared memory.
bool encode_bytes_2d(CUtensorMap *map, const void *base, int rows, int k, int box_rows, bool from_hbm)
{
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn)
        return false;
    const cuuint64_t gdim[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t gstride[1] = {(cuuint64_t)k};
    const cuuint32_t box[2] = {128u, (cuuint32_t)box_rows};
    const cuuint32_t estride[2] = {1u, 1u};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, from_hbm ? CU_TENSOR_MAP_L2_PROMOTION_L2_256B : CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// Token blocks that the matrix kernel is built for, and the one for n tokens in tb blocks of 64.
constexpr int kTokenBlocks[4] = {16, 32, 48, 64};

static int token_block(int tb, int n)
{
    for (int i = 0; tb == 1 && i < 3; ++i)
        if (n <= kTokenBlocks[i])
            return i;
    return 3;
}

// What the kernels of one chunk hand to each other.
struct Workspaces {
    int blocks = 0;              // blocks of 64 tokens they hold: one, or kTB
    float *x = nullptr, *qkv = nullptr, *q = nullptr, *h13 = nullptr;
    float *parts = nullptr;      // [kMaxParts][blocks * 64][dim]: partial row sums of Wo / W2, or the attention's key ranges
    int8_t *limbs = nullptr;
    float2 *ux = nullptr;
    float *ssq = nullptr;        // [blocks][groups / 4][64]
    CUtensorMap map_b_dim[4], map_b_hidden[4];   // by size of the token block: kTokenBlocks
    char *mem = nullptr;         // all of them
};

struct Prefill : Workspaces {
    PrefillModel m;
    cudaStream_t stream = nullptr;   // where all work on the buffers goes, their clearing included
    int kv_dim = 0, qkv_ld = 0, sms = 0;
    std::vector<CUtensorMap> maps;   // [layer][PF_W_COUNT]
    int *tokens = nullptr;
    int token_cap = 0;
    size_t attn_smem = 0;
    std::vector<void *> owned;
    unsigned long long launches = 0;
    // concurrent sequences
    int n_seq = 0, seq_len_b = 0;
    float *bkc = nullptr, *bvc = nullptr;      // [sequence][layer][kv_head][seq_len_b][head]
    int *meta = nullptr;                       // device: tokens[64], positions[64], sequences[64], arg-max[64]
    uint32_t *xn = nullptr;                    // [3][64][dim] bf16: the classifier's input in three pieces
    CUtensorMap map_xn;
    float *logits = nullptr;                   // [64][vocab]
    int *meta_host = nullptr;                  // pinned, 4 x 64
    float *logits_host = nullptr;              // pinned, [64][vocab]
    std::map<int, cudaGraphExec_t> step_graphs; // captured step per entry count
    unsigned long long step_launches = 0;
    bool step_ready = false;                    // all of the buffers of a step exist
    bool no_graph = false;
};

bool prefill_supported(const PrefillModel &m)
{
    const int kv_dim = m.n_kv_heads * m.head;
    return m.dim % 256 == 0 && m.hidden % 256 == 0 && kv_dim % kTileM == 0 && m.dim <= kMaxDim && m.hidden <= kMaxDim &&
           (m.head == 64 || m.head == 128) && m.n_heads * m.head == m.dim && m.n_layers > 0;
}

void prefill_destroy(Prefill *pf)
{
    if (!pf)
        return;
    for (auto &g : pf->step_graphs)
        cudaGraphExecDestroy(g.second);
    if (pf->meta_host)
        cudaFreeHost(pf->meta_host);
    if (pf->logits_host)
        cudaFreeHost(pf->logits_host);
    for (void *p : pf->owned)
        cudaFree(p);
    delete pf;
}

// Cleared on the stream of the kernels that use it: that stream does not wait for the default stream.
template <typename T>
static cudaError_t pf_alloc(Prefill *pf, T **out, size_t count)
{
    void *p = nullptr;
    cudaError_t e = alloc_fails(pf->m.fail_alloc) ? cudaErrorMemoryAllocation : cudaMalloc(&p, count * sizeof(T));
    if (e != cudaSuccess)
        return e;
    pf->owned.push_back(p);
    *out = static_cast<T *>(p);
    return cudaMemsetAsync(p, 0, count * sizeof(T), pf->stream);
}

static void pf_free(Prefill *pf, void *ptr)
{
    for (size_t i = 0; i < pf->owned.size(); ++i)
        if (pf->owned[i] == ptr) {
            cudaFree(ptr);
            pf->owned.erase(pf->owned.begin() + (long)i);
            return;
        }
}

template <typename T>
static cudaError_t pf_host_alloc(Prefill *pf, T **out, size_t count)
{
    return alloc_fails(pf->m.fail_alloc) ? cudaErrorMemoryAllocation
                                         : cudaHostAlloc(reinterpret_cast<void **>(out), count * sizeof(T), cudaHostAllocDefault);
}

// Workspaces of `blocks` blocks in the place of those there are, which stay if the new ones do not fit.  A concurrent step
// and a prompt of at most 64 tokens need one block (35 MB at the 7B shape), the chunks of a longer prompt four (141 MB).
// The captured steps hold the old addresses: they are captured again when they are next asked for.  First prompt of a
// 2-layer model of the 7B shape, ms, with eight allocations of four blocks for every caller and with this: 37 tokens 2.6
// and 0.9, 700 tokens 3.9 and 2.4; 300 tokens behind 37 0.77 and 1.6.
static cudaError_t make_workspaces(Prefill *pf, int blocks)
{
    const PrefillModel &m = pf->m;
    const size_t kmax = m.dim > m.hidden ? m.dim : m.hidden, tokens = (size_t)blocks * kT;
    Workspaces w;
    w.blocks = blocks;
    // one allocation: the parts are walked once for its size and once for their addresses
    size_t at = 0;
    auto take = [&](auto *&part, size_t count) {
        if (w.mem)
            part = reinterpret_cast<std::remove_reference_t<decltype(part)>>(w.mem + at);
        at += (count * sizeof(*part) + 1023) & ~(size_t)1023;
    };
    auto walk = [&]() {
        at = 0;
        take(w.x, tokens * m.dim);
        take(w.qkv, tokens * pf->qkv_ld);
        take(w.q, tokens * m.dim);
        take(w.h13, kWideParts * tokens * 2 * m.hidden);
        take(w.parts, kMaxParts * tokens * (m.dim + 2 * m.n_heads));
        take(w.limbs, (size_t)blocks * kN * kmax);
        take(w.ux, (kmax / 256) * tokens);
        take(w.ssq, (kmax / 256) * tokens);
    };
    walk();
    cudaError_t e = pf_alloc(pf, &w.mem, at);
    if (e != cudaSuccess)
        return e;
    walk();
    for (int i = 0; i < 4; ++i) {
        const int cols = 3 * kTokenBlocks[i], rows = kTokenBlocks[i] == kT ? blocks * cols : cols;
        if (!encode_bytes_2d(&w.map_b_dim[i], w.limbs, rows, m.dim, cols, false) ||
            !encode_bytes_2d(&w.map_b_hidden[i], w.limbs, rows, m.hidden, cols, false))
            return cudaErrorNotSupported;
    }
    for (auto &g : pf->step_graphs)
        cudaGraphExecDestroy(g.second);
    pf->step_graphs.clear();
    pf_free(pf, pf->mem);
    static_cast<Workspaces &>(*pf) = w;
    return cudaSuccess;
}

// The workspaces for n tokens.  Where four blocks do not fit, one has to do: chunks of 64 tokens.
static cudaError_t ensure_workspaces(Prefill *pf, int n)
{
    const int want = n > kT ? kTB : 1;
    if (pf->blocks >= want)
        return cudaSuccess;
    cudaError_t e = make_workspaces(pf, want);
    if (e == cudaErrorMemoryAllocation && want > 1) {
        cudaGetLastError();
        e = pf->blocks > 0 ? cudaSuccess : make_workspaces(pf, 1);
    }
    return e;
}

cudaError_t prefill_create(Prefill **out, const PrefillModel &m, cudaStream_t st, int n)
{
    *out = nullptr;
    if (!prefill_supported(m) || (int)m.layers.size() != m.n_layers)
        return cudaErrorInvalidValue;
    Prefill *pf = new Prefill();
    pf->m = m;
    pf->stream = st;
    pf->kv_dim = m.n_kv_heads * m.head;
    pf->qkv_ld = m.dim + 2 * pf->kv_dim;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&pf->sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = ensure_workspaces(pf, n);
    if (e != cudaSuccess) {
        prefill_destroy(pf);
        return e;
    }
    const int rows[PF_W_COUNT] = {m.dim, pf->kv_dim, pf->kv_dim, m.dim, m.hidden, m.hidden, m.dim};
    const int ks[PF_W_COUNT] = {m.dim, m.dim, m.dim, m.dim, m.dim, m.dim, m.hidden};
    pf->maps.resize((size_t)m.n_layers * PF_W_COUNT);
    bool ok = true;
    for (int l = 0; l < m.n_layers && ok; ++l)
        for (int w = 0; w < PF_W_COUNT && ok; ++w)
            ok = encode_bytes_2d(&pf->maps[(size_t)l * PF_W_COUNT + w], m.layers[(size_t)l].w[w], rows[w], ks[w], kTileM, true);
    if (!ok) {
        prefill_destroy(pf);
        return cudaErrorNotSupported;
    }
    // (the limit belongs to the kernel on the device, not to this context: it covers every shape)
    auto limit = [](auto kernel, size_t bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); };
    e = limit(pf_gemm_kernel<16>, GemmCfg<16>::smem(kMaxDim / 256));
    if (e == cudaSuccess)
        e = limit(pf_gemm_kernel<32>, GemmCfg<32>::smem(kMaxDim / 256));
    if (e == cudaSuccess)
        e = limit(pf_gemm_kernel<48>, GemmCfg<48>::smem(kMaxDim / 256));
    if (e == cudaSuccess)
        e = limit(pf_gemm_kernel<64>, GemmCfg<64>::smem(kMaxDim / 256));
    pf->attn_smem = m.head == 128 ? attn_smem_bytes<128>() : attn_smem_bytes<64>();
    if (e == cudaSuccess)
        e = m.head == 128 ? cudaFuncSetAttribute(pf_attention_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pf->attn_smem)
                          : cudaFuncSetAttribute(pf_attention_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pf->attn_smem);
    if (e != cudaSuccess) {
        prefill_destroy(pf);
        return e;
    }
    *out = pf;
    return cudaSuccess;
}

namespace {

// Every kernel of this file waits for the one in front (griddepcontrol.wait) before it touches what that one wrote, and
// lets the next one start at its own start: set-up, the first weight tiles and the launch itself are hidden behind the
// kernel in front.  A kernel is complete only when all its blocks are, and each of them has waited, so whoever waits for
// it also waits for everything before it.  37 tokens behind 900 positions, 16 layers of the 7B shape: 3.69 -> 3.30 ms;
// a step of 4 long sequences 2.72 -> 2.48 ms.
template <typename... P, typename... A>
cudaError_t launch(Prefill *pf, cudaStream_t st, void (*kernel)(P...), dim3 grid, int threads, size_t smem, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pf->m.pdl ? 1 : 0;
    ++pf->launches;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// How the groups of a row are dealt to parts, for `tb` blocks of 64 tokens.
struct Splits {
    int o, w2, w13;
};

Splits splits_for(const Prefill *pf, int tb)
{
    const PrefillModel &m = pf->m;
    // matrices with few row tiles (Wo, W2: dim / 128) deal the groups of a row to several blocks
    auto few = [&](int groups) {
        int ks = 1;
        while (ks * 2 <= kMaxParts && (m.dim / kTileM) * tb * ks * 2 <= pf->sms && groups / (ks * 2) >= 2)
            ks *= 2;
        return ks;
    };
    // W1/W3 have more tiles than SMs or nearly so: the part count that needs the fewest rounds of groups
    // (QKV stays whole: three parts for its 96 tiles at the 7B shape gain nothing and cost the RoPE kernel two more reads)
    const int tiles = 2 * m.hidden / kTileM, groups = m.dim / 256, blocks = pf->sms / tb;
    int best = 1, best_cost = 1 << 30;
    for (int ks = 1; ks <= kWideParts && ks <= groups; ++ks) {
        const int cost = ((tiles * ks + blocks - 1) / blocks) * ((groups + ks - 1) / ks);
        if (cost < best_cost) {
            best_cost = cost;
            best = ks;
        }
    }
    return Splits{few(m.dim / 256), few(m.hidden / 256), best};
}

cudaError_t launch_gemm(Prefill *pf, cudaStream_t st, int layer, const int *w, int nw, int k, float *out, int ldc, const int *col0,
                        int ksplit, int tb, int nvalid, bool normed)
{
    const PrefillModel &m = pf->m;
    const int rows_of[PF_W_COUNT] = {m.dim, pf->kv_dim, pf->kv_dim, m.dim, m.hidden, m.hidden, m.dim};
    PfGemmParams p{};
    int tiles = 0;
    for (int i = 0; i < nw; ++i) {
        p.seg[i].hdr = m.layers[(size_t)layer].h[w[i]];
        p.seg[i].rows = rows_of[w[i]];
        p.seg[i].col0 = col0[i];
        tiles += rows_of[w[i]] / kTileM;
    }
    p.nseg = nw;
    p.groups = k / 256;
    p.tblocks = tb;
    p.ux = pf->ux;
    p.out = out;
    p.ldc = ldc;
    p.ksplit = ksplit;
    p.ssq = normed ? pf->ssq : nullptr;
    p.nssq = (k / 256 + kLimbWarps - 1) / kLimbWarps;
    p.n = k;
    p.nvalid = nvalid;
    p.timeout_us = m.timeout_us;
    p.status = m.status;
    const CUtensorMap *base = &pf->maps[(size_t)layer * PF_W_COUNT];
    const CUtensorMap &a0 = base[w[0]], &a1 = base[w[nw > 1 ? 1 : 0]], &a2 = base[w[nw > 2 ? 2 : 0]];
    const int t = token_block(tb, nvalid);
    const CUtensorMap &b = k == m.dim ? pf->map_b_dim[t] : pf->map_b_hidden[t];
    const int per_block = pf->sms / tb;      // thread blocks per block of tokens
    const int grid = tb * (tiles * ksplit < per_block ? tiles * ksplit : per_block);
    auto go = [&](auto kernel, size_t smem) { return launch(pf, st, kernel, dim3((unsigned)grid), kGemmThreads, smem, a0, a1, a2, b, p); };
    switch (kTokenBlocks[t]) {
    case 16: return go(pf_gemm_kernel<16>, GemmCfg<16>::smem(p.groups));
    case 32: return go(pf_gemm_kernel<32>, GemmCfg<32>::smem(p.groups));
    case 48: return go(pf_gemm_kernel<48>, GemmCfg<48>::smem(p.groups));
    default: return go(pf_gemm_kernel<64>, GemmCfg<64>::smem(p.groups));
    }
}

template <int MODE>
cudaError_t launch_limbs(Prefill *pf, cudaStream_t st, float *a, const float *b, const float *parts, int nparts, int lda, int n, int tb, int nvalid)
{
    PfLimbParams p{};
    p.a = a;
    p.b = b;
    p.parts = parts;
    p.nparts = nparts;
    p.head = pf->m.head;
    p.lda = lda;
    p.n = n;
    p.nvalid = nvalid;
    p.limbs = pf->limbs;
    p.ux = pf->ux;
    p.ssq = pf->ssq;
    p.tpad = tb * kT;
    p.tt = kTokenBlocks[token_block(tb, nvalid)];
    const dim3 grid((unsigned)(tb > 1 ? tb * kT : p.tt), (unsigned)((n / 256 + kLimbWarps - 1) / kLimbWarps));
    return launch(pf, st, pf_limbs_kernel<MODE>, grid, kLimbThreads, 0, p);
}

}  // namespace

#define PF_CK(x)                  \
    do {                          \
        cudaError_t e_ = (x);     \
        if (e_ != cudaSuccess)    \
            return e_;            \
    } while (0)

// Positions pos0 .. pos0 + n - 1 with the input tokens given (host pointer), enqueued on `st`.
cudaError_t prefill_run(Prefill *pf, cudaStream_t st, const int *tokens_host, int n, int pos0)
{
    const PrefillModel &m = pf->m;
    if (n > pf->token_cap) {
        int *t = nullptr;
        PF_CK(pf_alloc(pf, &t, (size_t)(n + kT)));
        pf->tokens = t;
        pf->token_cap = n;
    }
    PF_CK(cudaMemcpyAsync(pf->tokens, tokens_host, sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, st));
    PF_CK(ensure_workspaces(pf, n));
    const int dim = m.dim, hidden = m.hidden, kvd = pf->kv_dim, chunk = pf->blocks * kT;
    for (int c0 = 0; c0 < n; c0 += chunk) {
        const int nv = n - c0 < chunk ? n - c0 : chunk;
        const int tb = (nv + kT - 1) / kT;
        const Splits ks = splits_for(pf, tb);
        pf_embed_kernel<<<tb * kT, 256, 0, st>>>(pf->tokens + c0, nv, m.emb, dim, m.vocab, pf->x);    // behind a copy or a whole chunk
        ++pf->launches;
        PF_CK(cudaGetLastError());
        int pending = 0;     // partial row sums in `parts` that the next RMSNorm adds to x
        for (int l = 0; l < m.n_layers; ++l) {
            const PrefillLayerDesc &L = m.layers[(size_t)l];
            PF_CK(launch_limbs<PF_IN_NORM>(pf, st, pf->x, L.rms_att, pf->parts, pending, dim, dim, tb, nv));
            {
                const int w[3] = {PF_WQ, PF_WK, PF_WV}, col0[3] = {0, dim, dim + kvd};
                PF_CK(launch_gemm(pf, st, l, w, 3, dim, pf->qkv, pf->qkv_ld, col0, 1, tb, nv, true));
            }
            {
                PfRopeParams r{};
                r.qkv = pf->qkv; r.q = pf->q; r.k_cache = L.kc; r.v_cache = L.vc;
                r.rope_cos = m.rope_cos; r.rope_sin = m.rope_sin;
                r.dim = dim; r.kv_dim = kvd; r.head = m.head; r.seq_len = m.seq_len; r.pos0 = pos0 + c0; r.nvalid = nv;
                r.nparts = 1;
                const dim3 grid((unsigned)(tb * kT), (unsigned)((pf->qkv_ld / 2 + 255) / 256));
                PF_CK(launch(pf, st, pf_rope_kv_kernel, grid, 256, 0, r));
            }
            int nsplit = 1;
            {
                // Key ranges per (head, 128 queries): the count that needs the fewest rounds of key tiles with one block per
                // SM; a block's set-up (the pieces of Q, the first tile through every role) and the merge of its part cost
                // about three tiles.
                const int tiles = (pos0 + c0 + nv + kAttnKeys - 1) / kAttnKeys;
                const int base = m.n_heads * ((nv + kAttnQ - 1) / kAttnQ);
                int best = 0;
                for (int ns = 1; ns <= kMaxParts && ns <= tiles; ++ns) {
                    const int cost = ((base * ns + pf->sms - 1) / pf->sms) * ((tiles + ns - 1) / ns + 3);
                    if (ns == 1 || cost < best) {
                        best = cost;
                        nsplit = ns;
                    }
                }
                PfAttnParams a{};
                a.q = pf->q; a.k_cache = L.kc; a.v_cache = L.vc; a.parts = pf->parts;
                a.dim = dim; a.kv_mul = m.n_heads / m.n_kv_heads; a.seq_len = m.seq_len; a.pos0 = pos0 + c0; a.nvalid = nv;
                a.nsplit = nsplit; a.tpad = tb * kT; a.timeout_us = m.timeout_us; a.status = m.status;
                const dim3 grid((unsigned)m.n_heads, (unsigned)((nv + kAttnQ - 1) / kAttnQ), (unsigned)nsplit);
                PF_CK(launch(pf, st, m.head == 128 ? pf_attention_kernel<128> : pf_attention_kernel<64>, grid, kAttnThreads, pf->attn_smem, a));
            }
            PF_CK(launch_limbs<PF_IN_ATTN>(pf, st, nullptr, nullptr, pf->parts, nsplit, dim, dim, tb, nv));
            {
                const int w[1] = {PF_WO}, col0[1] = {0};
                PF_CK(launch_gemm(pf, st, l, w, 1, dim, pf->parts, dim, col0, ks.o, tb, nv, false));
            }
            PF_CK(launch_limbs<PF_IN_NORM>(pf, st, pf->x, L.rms_ffn, pf->parts, ks.o, dim, dim, tb, nv));
            {
                const int w[2] = {PF_W1, PF_W3}, col0[2] = {0, hidden};
                PF_CK(launch_gemm(pf, st, l, w, 2, dim, pf->h13, 2 * hidden, col0, ks.w13, tb, nv, true));
            }
            PF_CK(launch_limbs<PF_IN_SWIGLU>(pf, st, pf->h13, pf->h13 + hidden, nullptr, ks.w13, 2 * hidden, hidden, tb, nv));
            {
                const int w[1] = {PF_W2}, col0[1] = {0};
                PF_CK(launch_gemm(pf, st, l, w, 1, hidden, pf->parts, dim, col0, ks.w2, tb, nv, false));
            }
            pending = ks.w2;
        }
    }
    return cudaSuccess;
}

// Caches for n_seq sequences of seq_len positions each (replaces an earlier set).
cudaError_t prefill_batch_create(Prefill *pf, int n_seq, int seq_len)
{
    const PrefillModel &m = pf->m;
    if (n_seq < 1 || seq_len < 1 || seq_len > m.seq_len)
        return cudaErrorInvalidValue;
    const size_t per_seq = (size_t)m.n_layers * m.n_kv_heads * seq_len * m.head;
    for (auto &g : pf->step_graphs)
        cudaGraphExecDestroy(g.second);
    pf->step_graphs.clear();
    if (pf->bkc) {
        pf_free(pf, pf->bkc);
        pf_free(pf, pf->bvc);
        pf->bkc = pf->bvc = nullptr;
        pf->n_seq = 0;
    }
    PF_CK(pf_alloc(pf, &pf->bkc, per_seq * n_seq));
    PF_CK(pf_alloc(pf, &pf->bvc, per_seq * n_seq));
    if (!pf->step_ready) {      // what an earlier call that failed half-way made is there already
        if (!pf->meta)
            PF_CK(pf_alloc(pf, &pf->meta, (size_t)4 * kT));
        if (!pf->xn)
            PF_CK(pf_alloc(pf, &pf->xn, (size_t)kN * m.dim / 2));
        if (!encode_bytes_2d(&pf->map_xn, pf->xn, kN, 2 * m.dim, kN, false))
            return cudaErrorNotSupported;
        if (!pf->logits)
            PF_CK(pf_alloc(pf, &pf->logits, (size_t)kT * m.vocab));
        if (!pf->meta_host)
            PF_CK(pf_host_alloc(pf, &pf->meta_host, (size_t)4 * kT));
        if (!pf->logits_host)
            PF_CK(pf_host_alloc(pf, &pf->logits_host, (size_t)kT * m.vocab));
        PF_CK(cudaFuncSetAttribute(bd_classifier_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kClsStages * kClsStage + 1024));
        pf->step_ready = true;
    }
    pf->n_seq = n_seq;
    pf->seq_len_b = seq_len;
    return cudaSuccess;
}

// One decode step of n <= 64 (sequence, position, token) triples on one sweep over the weights; a sequence
// may appear several times with different positions (their K/V rows are all written before the attention).
// logits_out [n][vocab] and argmax_out [n] are host pointers (either may be null); blocks until done.
// Everything one step of n entries puts on the stream: tokens / positions / sequences in, all layers, classifier,
// arg-max ids out (pinned buffers on both ends, so the whole step can be captured into a graph).
static cudaError_t batch_enqueue(Prefill *pf, cudaStream_t st, int nv)
{
    const PrefillModel &m = pf->m;
    const int dim = m.dim, hidden = m.hidden, kvd = pf->kv_dim;
    PF_CK(cudaMemcpyAsync(pf->meta, pf->meta_host, sizeof(int) * 3 * kT, cudaMemcpyHostToDevice, st));
    const int *d_tok = pf->meta, *d_pos = pf->meta + kT, *d_seq = pf->meta + 2 * kT;
    int *d_arg = pf->meta + 3 * kT;
    const long long layer_stride = (long long)m.n_kv_heads * pf->seq_len_b * m.head;
    const long long seq_stride = layer_stride * m.n_layers;
    pf_embed_kernel<<<kT, 256, 0, st>>>(d_tok, nv, m.emb, dim, m.vocab, pf->x);      // behind a copy
    ++pf->launches;
    PF_CK(cudaGetLastError());
    int pending = 0;
    const Splits ks = splits_for(pf, 1);
    const int nsplit = bd_splits(m.n_heads, nv, pf->sms);
    for (int l = 0; l < m.n_layers; ++l) {
        const PrefillLayerDesc &L = m.layers[(size_t)l];
        PF_CK(launch_limbs<PF_IN_NORM>(pf, st, pf->x, L.rms_att, pf->parts, pending, dim, dim, 1, nv));
        {
            const int w[3] = {PF_WQ, PF_WK, PF_WV}, col0[3] = {0, dim, dim + kvd};
            PF_CK(launch_gemm(pf, st, l, w, 3, dim, pf->qkv, pf->qkv_ld, col0, 1, 1, nv, true));
        }
        {
            PfRopeParams r{};
            r.qkv = pf->qkv; r.q = pf->q; r.k_cache = pf->bkc + l * layer_stride; r.v_cache = pf->bvc + l * layer_stride;
            r.rope_cos = m.rope_cos; r.rope_sin = m.rope_sin;
            r.dim = dim; r.kv_dim = kvd; r.head = m.head; r.seq_len = pf->seq_len_b; r.pos0 = 0; r.nvalid = nv;
            r.nparts = 1;
            r.pos_of = d_pos; r.seq_of = d_seq; r.seq_stride = seq_stride;
            const dim3 grid((unsigned)kT, (unsigned)((pf->qkv_ld / 2 + 255) / 256));
            PF_CK(launch(pf, st, pf_rope_kv_kernel, grid, 256, 0, r));
        }
        {
            BdAttnParams a{};
            a.q = pf->q; a.k_cache = pf->bkc + l * layer_stride; a.v_cache = pf->bvc + l * layer_stride; a.seq_stride = seq_stride;
            a.pos_of = d_pos; a.seq_of = d_seq; a.parts = pf->parts;
            a.dim = dim; a.kv_mul = m.n_heads / m.n_kv_heads; a.seq_len = pf->seq_len_b; a.nvalid = nv;
            a.nsplit = nsplit;
            const dim3 grid((unsigned)m.n_heads, (unsigned)nv, (unsigned)nsplit);
            PF_CK(launch(pf, st, m.head == 128 ? bd_attention_kernel<128> : bd_attention_kernel<64>, grid, kBdThreads, 0, a));
        }
        PF_CK(launch_limbs<PF_IN_ATTN>(pf, st, nullptr, nullptr, pf->parts, nsplit, dim, dim, 1, nv));
        {
            const int w[1] = {PF_WO}, col0[1] = {0};
            PF_CK(launch_gemm(pf, st, l, w, 1, dim, pf->parts, dim, col0, ks.o, 1, nv, false));
        }
        PF_CK(launch_limbs<PF_IN_NORM>(pf, st, pf->x, L.rms_ffn, pf->parts, ks.o, dim, dim, 1, nv));
        {
            const int w[2] = {PF_W1, PF_W3}, col0[2] = {0, hidden};
            PF_CK(launch_gemm(pf, st, l, w, 2, dim, pf->h13, 2 * hidden, col0, ks.w13, 1, nv, true));
        }
        PF_CK(launch_limbs<PF_IN_SWIGLU>(pf, st, pf->h13, pf->h13 + hidden, nullptr, ks.w13, 2 * hidden, hidden, 1, nv));
        {
            const int w[1] = {PF_W2}, col0[1] = {0};
            PF_CK(launch_gemm(pf, st, l, w, 1, hidden, pf->parts, dim, col0, ks.w2, 1, nv, false));
        }
        pending = ks.w2;
    }
    PF_CK(launch(pf, st, bd_final_norm_kernel, dim3((unsigned)kT), 256, 0, pf->x, pf->parts, pending, m.rms_final, dim, nv, pf->xn));
    {
        BdClsParams c{};
        c.wcls = m.wcls; c.vocab = m.vocab; c.dim = dim; c.nvalid = nv; c.logits = pf->logits;
        c.timeout_us = m.timeout_us; c.status = m.status;
        const int tiles = (m.vocab + kClsRows - 1) / kClsRows;
        PF_CK(launch(pf, st, bd_classifier_kernel, dim3((unsigned)(tiles < pf->sms ? tiles : pf->sms)), kClsThreads,
                     (size_t)(kClsStages * kClsStage + 1024), pf->map_xn, c));
    }
    PF_CK(launch(pf, st, bd_argmax_kernel, dim3((unsigned)nv), 256, 0, pf->logits, m.vocab, nv, d_arg));
    PF_CK(cudaMemcpyAsync(pf->meta_host + 3 * kT, d_arg, sizeof(int) * kT, cudaMemcpyDeviceToHost, st));
    return cudaSuccess;
}

cudaError_t prefill_batch_forward(Prefill *pf, cudaStream_t st, const int *tokens, const int *pos, const int *seq, int n, float *logits_out,
                                  int *argmax_out)
{
    const PrefillModel &m = pf->m;
    const int nv = n;
    for (int i = 0; i < kT; ++i) {
        pf->meta_host[i] = i < n ? tokens[i] : 0;
        pf->meta_host[kT + i] = i < n ? pos[i] : 0;
        pf->meta_host[2 * kT + i] = i < n ? seq[i] : 0;
    }
    // The step is about 330 launches of kernels that mostly run for a few microseconds: replayed as one graph per
    // entry count (grids and parameters depend on it; the caches and buffers stay where they are until
    // prefill_batch_create runs again).
    cudaGraphExec_t exec = nullptr;
    auto it = pf->step_graphs.find(nv);
    if (it != pf->step_graphs.end()) {
        exec = it->second;
    } else if (!pf->no_graph) {
        cudaGraph_t graph = nullptr;
        const unsigned long long before = pf->launches;
        if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
            const cudaError_t ce = batch_enqueue(pf, st, nv);
            const cudaError_t ee = cudaStreamEndCapture(st, &graph);
            if (ce == cudaSuccess && ee == cudaSuccess && graph && cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess) {
                pf->step_graphs[nv] = exec;
                pf->step_launches = pf->launches - before;
            } else {
                exec = nullptr;
                pf->no_graph = true;      // direct launches from now on
                cudaGetLastError();
            }
            if (graph)
                cudaGraphDestroy(graph);
        } else {
            pf->no_graph = true;
            cudaGetLastError();
        }
        pf->launches = before;
    }
    if (exec) {
        PF_CK(cudaGraphLaunch(exec, st));
        pf->launches += pf->step_launches;
    } else {
        PF_CK(batch_enqueue(pf, st, nv));
    }
    if (logits_out)
        PF_CK(cudaMemcpyAsync(pf->logits_host, pf->logits, sizeof(float) * (size_t)nv * m.vocab, cudaMemcpyDeviceToHost, st));
    PF_CK(cudaStreamSynchronize(st));
    if (logits_out)
        memcpy(logits_out, pf->logits_host, sizeof(float) * (size_t)nv * m.vocab);
    if (argmax_out)
        for (int i = 0; i < n; ++i)
            argmax_out[i] = pf->meta_host[3 * kT + i];
    return cudaSuccess;
}

int prefill_batch_sequences(const Prefill *pf)
{
    return pf ? pf->n_seq : 0;
}

int prefill_batch_seq_len(const Prefill *pf)
{
    return pf ? pf->seq_len_b : 0;
}

unsigned long long prefill_launches(const Prefill *pf)
{
    return pf ? pf->launches : 0;
}

}  // namespace l2j
