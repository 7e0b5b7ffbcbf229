// fused_layers_kernel: every layer of a token in ONE persistent launch (sm_100a).
//
// The per-step kernels of l2j_kernels.cu stream at HBM speed but pay a start-up chain at each of
// their five boundaries per layer: a block holds nearly all of an SM's shared memory, so the next
// kernel's block cannot become resident, let alone prefetch, before the one in front has left.
// Here the blocks never leave.  One block per SM; its warps keep their roles for the whole token:
//
//   producer thread   walks the fixed sequence of stages of this block (layer by layer: QKV rows,
//                     cached K/V rows of the attention step, Wo rows, W1/W3 row pairs, W2 rows) and
//                     streams them with bulk copies (TMA engine) into ONE shared-memory byte ring,
//                     as far ahead as the ring has room.  Weights and old cache rows never depend
//                     on this token's activations, so while the consumers wait at a phase boundary
//                     the ring fills with the next phase: HBM does not idle.
//   consumer warps    per phase: poll the input vector, which arrives as (value, tag) pairs, RMSNorm,
//                     fixed-point limbs, then dp4a over the block's stages as they land.
//   epilogue warp     adds the per-warp partial sums of a group of stages, applies RoPE + cache write,
//                     residual add or SwiGLU, and hands every result on as a pair.
//
// Stages are dealt to the blocks round-robin, continuing across phases, so every block streams the
// same number of bytes per token (+- one stage).  The attention step's units (head, 32 positions)
// are dealt in contiguous runs; a block folds the units of one head into one partial (m, l, o), and the block with the
// head's first positions merges the few partials of the head (at most kAttSlots) in a fixed order.
//
// What bounds it (7B shape, position 160): a layer takes 44 us where its bytes take 31.5 at the measured copy rate.  The
// ring holds 4.4 us of a block's share of the HBM; a boundary between two phases costs 2 to 3 us from the median block's last
// result to the next block's first dot product, and the attention step and Wo, which hardly stream, 11 us together.  Two rows per warp
// with half as many elements each leave registers to fetch the next stage's bytes while the dot products of this one run; 14
// consumer warps because more than 16 warps would have fewer than 128 registers and spill, which costs more than it saves here.
// Against counters between the blocks, 18 warps with a row each and a merge of the attention partials in every block: 48 greedy
// forwards of 7B 88.6 -> 69 to 72 ms (by machine), 8 steps behind 3840 positions 22.4 -> 17.7 to 18.5; 24 forwards of 13B, per-step
// kernels before, 70.2 -> 62.7 to 65.9.
//
// Blocks wait for each other, so all of them must be resident: the grid is one block per SM and the launch is
// cooperative.  Every wait is bounded by the SM's cycle counter.  A hand-over between blocks that runs out raises
// L2J_DS_WAIT_TIMEOUT in the status word, and every hand-over that any warp of the block still waits for gives up after 2 us;
// the block then still works through all of its stages with the (wrong) inputs it has, so that producer, consumers and epilogue warp
// stay in step and no bulk copy is in flight when the block ends.
//
// Reference counterparts (paths relative to src/main/java/com/lastbot/llama2j/): the layer body of
// Run.java:418-508 with kernel/MatMul.java:360-444, RootMeanSquare.java:78-118,
// WeightNormalizeAndScale.java:191-239, ApplyRope.java:144-182, AttentionLoop.java:116-164,
// ExpSumNormalize.java:82-131, AccumWeightedValue.java:148-173, Accum.java:70-83, Silu.java:118-135.

#include "l2j_device.cuh"
#include "l2j_internal.h"

#include <cfloat>
#include <cmath>

#define L2J_DS_WAIT_TIMEOUT 0x1
#define L2J_LATE_INPUT 0x1
#define L2J_LATE_ROWS 0x2
#define L2J_LATE_PARTIALS 0x4
#define L2J_LATE_RESIDUAL 0x8

namespace l2j {

static_assert(sizeof(FusedParams) <= 4000, "the parameter block must fit the kernel parameter space");

namespace {

constexpr int kFDesc = 16;              // stage descriptors (and full/empty barrier pairs) in flight
constexpr int kFRedBufs = 4;
constexpr int kFGroup = 4;               // stages of a block that are folded and handed to the epilogue warp together
constexpr int kFBarFull = 0;            // uint64 full[16]
constexpr int kFBarEmpty = 128;         // uint64 empty[16]
constexpr int kFBarRedFull = 256;       // uint64 red_full[4]
constexpr int kFBarRedEmpty = 288;      // uint64 red_empty[4]
constexpr int kFVStart = 328;           // int vstart[16]: the producer's bookkeeping of where each stage in flight begins
constexpr int kFScratch = 392;          // float scratch[14]
constexpr int kFLost = 448;             // int: a wait of the block has run out, or one of an earlier forward had
constexpr int kFLate = 452;             // int: the L2J_LATE_* bits
constexpr int kFDescOff = 512;          // FStage desc[16]
constexpr int kFRedOff = 1024;          // 4 x 112 floats: [stage of the group][row of the stage][warp of the row]
constexpr int kFRedStride = 4 * kFGroup * 2 * kFusedConsWarps;   // a stage has two rows per set of warps
constexpr int kFRopeOff = 3328;         // float cos[64], sin[64] of the token's position
constexpr int kFInvTab = 3840;          // float inv[64]: value of one fixed-point unit of each group of the input vector
constexpr int kFHeader = kFusedHeaderBytes;   // end of the fixed part (128-byte aligned)
static_assert(kFScratch + 4 * kFusedConsWarps <= kFLost && kFLate + 4 <= kFDescOff && kFRedOff + kFRedBufs * kFRedStride <= kFRopeOff, "header layout");
static_assert(kFInvTab + 4 * (kFusedMaxRow / 256) <= kFHeader, "header layout");
constexpr int kFCons = kFusedConsWarps * 32;
constexpr int kAttBatch = 4;            // cached positions that a lane group works on at a time
constexpr uint64_t kFShortWaitNs = 2000;
constexpr int kFLateTag = 0x40000000;   // what a reader's tag is off by while l2j_debug_late makes it wait for nothing

struct FStage {
    int off, nrows, e0a, e0b;   // what the consumers of a matrix stage need, in one 16-byte load: byte offset in the
                                // ring, rows, element offset of the first row of each half relative to the headers
    int seg, row0, aux, pad;
    // attention stage: seg = head, row0 = first position, nrows = positions (newest included),
    // e0a = positions that travel through the ring (older than the token), aux = byte offset of the V rows
};

__device__ __forceinline__ uint4 lds_v4(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

__device__ __forceinline__ float2 lds_f2(uint32_t addr)
{
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}

__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c)
{
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// Two (value, sequence number) pairs of the hand-over between blocks, from L2.
__device__ __forceinline__ float4 ld_pairs2_gpu(const float2 *p)
{
    float4 v;
    asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ float2 ld_pair_gpu(const float2 *p)
{
    float2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
    return v;
}

// An exchange and not a store: a plain store waits in the SM behind the stream, an atomic goes at once (7B shape, W2 -> QKV: the
// input vector is complete 3.7 instead of 6.5 us after the median block's last result).
__device__ __forceinline__ void st_pair_gpu(float2 *p, float v, int tag)
{
    unsigned long long old;
    asm volatile("atom.relaxed.gpu.global.exch.b64 %0, [%1], %2;"
                 : "=l"(old)
                 : "l"(p), "l"(((unsigned long long)(unsigned int)tag << 32) | __float_as_uint(v))
                 : "memory");
}

__device__ __forceinline__ bool tagged(const float4 &v, int tag)
{
    return __float_as_int(v.y) == tag && __float_as_int(v.w) == tag;
}

// The block's word for "a wait has run out": whichever warp it was, every hand-over that the block still waits for gives up early.
__device__ __forceinline__ void set_block_lost(uint32_t sbase)
{
    asm volatile("st.volatile.shared.s32 [%0], 1;" ::"r"(sbase + kFLost) : "memory");
}

// A reader's tag: the one it waits for, or one that nobody writes while l2j_debug_late says so.
__device__ __forceinline__ int reader_tag(uint32_t sbase, int tag, int reader)
{
    int late;
    asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(late) : "r"(sbase + kFLate) : "memory");
    return late & reader ? tag ^ kFLateTag : tag;
}

__device__ __forceinline__ bool block_lost(uint32_t sbase)
{
    int v;
    asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(v) : "r"(sbase + kFLost) : "memory");
    return v != 0;
}

// Has a hand-over that the block waits for since c0 run out?
__device__ __forceinline__ bool hand_over_lost(uint32_t sbase, long long c0, uint64_t wait_ns)
{
    return sm_clock() - c0 > (long long)(2 * (block_lost(sbase) ? kFShortWaitNs : wait_ns));
}

// Bulk copy without a cache hint (cached K/V rows are read again by the next token).
__device__ __forceinline__ void bulk_g2s_plain(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}

template <int RT, int STEP>
struct Fold {
    static __device__ __forceinline__ float run(const float (&v)[RT], int lane)
    {
        if constexpr (RT == 1) {
            float k = v[0];
#pragma unroll
            for (int o = STEP; o > 0; o >>= 1)
                k += __shfl_xor_sync(0xffffffffu, k, o);
            return k;
        } else {
            constexpr int H = RT / 2;
            const bool up = (lane & STEP) != 0;
            float k[H];
#pragma unroll
            for (int i = 0; i < H; ++i) {
                const float keep = up ? v[H + i] : v[i];
                const float send = up ? v[i] : v[H + i];
                k[i] = keep + __shfl_xor_sync(0xffffffffu, send, STEP);
            }
            return Fold<H, STEP / 2>::run(k, lane);
        }
    }
};

// How the attention step of a token at position `pos` is dealt to the blocks: units of (head, chunk of
// kAttChunk positions), head-major, in contiguous runs over the first `ga` blocks.
struct AttSplit {
    int nchunk, units, ga;
};

__device__ __forceinline__ AttSplit att_split(const FusedParams &P, int pos, int grid)
{
    AttSplit a;
    a.nchunk = (pos + kAttChunk) / kAttChunk;   // ceil((pos + 1) / chunk)
    a.units = P.n_heads * a.nchunk;
    // Short contexts are a matter of latency, not bandwidth: three blocks per head keep the partials of a head
    // few enough (four) for the step behind to fetch them in one round of loads.
    const int per_head = a.nchunk <= 512 / kAttChunk ? 3 : kAttMaxSplit;
    a.ga = min(min(grid, P.n_heads * per_head), a.units);
    return a;
}

// (32-bit divisions: units * blocks stays below 2^31 for every head count and sequence length that fits a device.)
__device__ __forceinline__ int att_first_unit(const AttSplit &a, int b)
{
    return (int)((unsigned int)b * (unsigned int)a.units / (unsigned int)a.ga);
}

__device__ __forceinline__ int att_block_of(const AttSplit &a, int u)
{
    return (int)(((unsigned int)(u + 1) * (unsigned int)a.ga + (unsigned int)a.units - 1u) / (unsigned int)a.units) - 1;
}

// Partial results of head h.
__device__ __forceinline__ int att_partials(const AttSplit &a, int h)
{
    return att_block_of(a, (h + 1) * a.nchunk - 1) - att_block_of(a, h * a.nchunk) + 1;
}

// Stage index -> (segment, first row, row count) of a ring phase.
__device__ __forceinline__ void stage_rows(const MvParams &p, int s, int &seg, int &row0, int &nrows)
{
    seg = 0;
    if (!p.paired && p.nseg > 1) {
        if (s >= p.seg_stages[0]) {
            s -= p.seg_stages[0];
            seg = 1;
            if (s >= p.seg_stages[1]) {
                s -= p.seg_stages[1];
                seg = 2;
            }
        }
    }
    row0 = s * p.rs;
    nrows = min(p.rs, p.seg[seg].rows - row0);
}

__device__ __forceinline__ int first_stage_of(int b, int rot, int grid)
{
    int f = b - rot;
    return f < 0 ? f + grid : f;
}

__device__ __forceinline__ void fused_trace(const FusedParams &P, int phase_index, int k)
{
    if (P.trace)
        P.trace[((int64_t)blockIdx.x * (5 * P.n_layers) + phase_index) * 8 + k] = (unsigned long long)global_timer_ns();
}

// -------------------------------------------------------------------------------------------------
// producer
// -------------------------------------------------------------------------------------------------

struct Producer {
    uint8_t *smem;
    uint32_t sbase, ring_base;
    int vhead;              // bytes handed out since the last rebase()
    int off;                // vhead's position in the ring
    int ring_bytes;
    int seq, tail;          // descriptors issued / known to be released
    int vtail;              // where the oldest stage not known to be released begins
    uint64_t wait_ns;
    int pos;                // the token's position, -1 until the kernel in front has set it
    AttSplit as;

    // Room for `bytes` contiguous bytes and a free descriptor; returns the offset in the ring.
    __device__ __forceinline__ uint32_t acquire(uint32_t bytes)
    {
        int *vstart = reinterpret_cast<int *>(smem + kFVStart);
        if (off + (int)bytes > ring_bytes) {
            vhead += ring_bytes - off;
            off = 0;
        }
        const int vend = vhead + (int)bytes;
        while (tail < seq && (seq - tail >= kFDesc || vend - ring_bytes > vtail)) {
            if (!mbar_wait_bounded(sbase + kFBarEmpty + 8 * (tail % kFDesc), (uint32_t)(tail / kFDesc) & 1u,
                                   wait_ns))
                set_block_lost(sbase);
            ++tail;
            vtail = vstart[tail % kFDesc];
        }
        if (tail == seq)
            vtail = vhead;
        vstart[seq % kFDesc] = vhead;
        const uint32_t at = (uint32_t)off;
        const int step = (int)((bytes + 127u) & ~127u);
        vhead += step;
        off += step;
        return at;
    }

    // Counts from the oldest stage in flight on.  Grouped heads that share a long cache take a block's ring through more than 2^31
    // bytes in one token.  (48 forwards of 7B: 68.65 ms without it, 68.90 with it; with a
    // difference modulo 2^32 in acquire() 0.5 ms more than without.)
    __device__ __forceinline__ void rebase(int lane)
    {
        int *vstart = reinterpret_cast<int *>(smem + kFVStart);
        const int base = tail < seq ? vtail : vhead;
        __syncwarp(0xfu);
        for (int i = tail + lane; i < seq; i += 4)
            vstart[i % kFDesc] -= base;
        __syncwarp(0xfu);
        vhead -= base;
        vtail = 0;
    }
};
constexpr int kFRebase = 1 << 30;       // looked at once per layer and attention unit: neither adds as much again

__device__ __forceinline__ void producer_learn_pos(Producer &pr, const FusedParams &P, int grid)
{
    if (pr.pos < 0) {
        // The position is set by the kernel in front; everything touched so far was weights.
        pdl_wait();
        pr.pos = __ldcg(&P.state->cur_pos);
        pr.as = att_split(P, pr.pos, grid);
    }
}

// The producer is the first four lanes of its warp.  All four keep the same bookkeeping; a stage's (up to) four
// bulk copies (rows of one or two matrices, their group headers) are one instruction stream with per-lane
// operands: lane = 2 * is_header + half.  Every lane arrives on the stage's barrier with the bytes of its own
// copy (the barrier counts four arrivals), so the lanes need not talk to each other.
//
// The block's stages of a phase: first, first + G, ...  One pass of the inner loop is the producer's time per stage, and the
// ring cannot be drained faster than that, so everything that does not change from stage to stage is set up per
// phase and segment, and positions advance by additions in units of quantisation groups.
__device__ __forceinline__ void produce_phase(Producer &pr, const FusedParams &P, const MvParams &p, int k, int layer, int first, int G,
                                              uint64_t pol, int lane)
{
    const int h = lane & 1, is_hdr = lane >> 1;
    const int paired = p.paired, rs = p.rs, groups = p.n >> 8, S = p.total_stages;
    const bool copy = (paired || h == 0) && !(P.debug_no_copy & 1);
    const uint32_t slot_bytes = (uint32_t)p.slot_bytes;
    const uint32_t dst0 = pr.ring_base + (is_hdr ? (uint32_t)(p.hdr_off + h * p.half_hdr) : (uint32_t)(h * rs * p.n));   // h is 0 or the stage is paired
    const int unit = is_hdr ? 8 : 256;
    const uint32_t desc0 = pr.sbase + kFDescOff;
    int s = first, s0 = 0, seg = 0;
    while (s < S) {
        while (!paired && seg < 2 && s >= s0 + p.seg_stages[seg]) {
            s0 += p.seg_stages[seg];
            ++seg;
        }
        const int s1 = paired ? S : s0 + p.seg_stages[seg];
        const MvSeg &sg = p.seg[paired ? h : seg];
        const uint8_t *src = is_hdr ? reinterpret_cast<const uint8_t *>(sg.hdr) : sg.payload;
        int left = sg.rows - (s - s0) * rs;                      // rows from the stage's first one on
        int gi = (int)((sg.flat0 + (int64_t)layer * P.seg_step[k][paired ? h : seg]) >> 8) + (s - s0) * rs * groups;   // its first group
        const int grs = G * rs, ggr = grs * groups;
        for (; s < s1; s += G, left -= grs, gi += ggr) {
            const int nrows = min(rs, left);
            const uint32_t off = pr.acquire(slot_bytes);
            const int e = pr.seq % kFDesc;
            const uint32_t full = pr.sbase + kFBarFull + 8 * e;
            const int ga = gi & ~1;                              // headers are copied from an even group on: 16-byte aligned
            const int ng = nrows * groups;
            const uint32_t bytes = (uint32_t)(is_hdr ? ((gi + ng + 1) & ~1) - ga : ng) * (uint32_t)unit;
            const int shift = (gi - ga) << 8;
            if (lane == 0)
                asm volatile("st.shared.v2.u32 [%0], {%1, %2};\n\tst.shared.u32 [%0 + 8], %3;" ::"r"(desc0 + 32u * (uint32_t)e), "r"(off),
                             "r"(nrows), "r"(shift)
                             : "memory");
            if (lane == 1)
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(desc0 + 32u * (uint32_t)e + 12u), "r"(shift) : "memory");
            if (copy) {
                mbar_arrive_expect_tx(full, bytes);
                bulk_g2s(dst0 + off, src + (int64_t)(is_hdr ? ga : gi) * unit, bytes, full, pol);
            } else {
                mbar_arrive(full);
            }
            ++pr.seq;
        }
    }
}

__device__ __forceinline__ void produce_att_stage(Producer &pr, const FusedParams &P, int layer, int unit, const AttSplit &a, int pos,
                                                  int lane)
{
    const int h = unit / a.nchunk, c = unit - h * a.nchunk;
    const int t0 = c * kAttChunk;
    const int cnt = min(pos + 1, t0 + kAttChunk) - t0;       // positions of the unit, the token's own included
    const int old = min(pos, t0 + kAttChunk) - t0;           // those that were cached by earlier tokens
    const uint32_t kbytes = (uint32_t)old * (uint32_t)P.head * 4u;
    const uint32_t voff = (kbytes + 127u) & ~127u;
    const uint32_t off = pr.acquire(2 * voff);
    const int e = pr.seq % kFDesc;
    const uint32_t full = pr.sbase + kFBarFull + 8 * e;
    FStage *desc = reinterpret_cast<FStage *>(pr.smem + kFDescOff) + e;
    const bool copy = old > 0 && !(P.debug_no_copy & 1) && lane < 2;
    if (lane == 0)
        *reinterpret_cast<int4 *>(desc) = make_int4((int)off, cnt, old, 0);
    if (lane == 1) {
        desc->seg = h;
        desc->row0 = t0;
        desc->aux = (int)voff;
    }
    if (copy) {      // lane 0 the K rows, lane 1 the V rows
        const int kvh = h / P.kv_mul;
        const int64_t row = ((int64_t)kvh * P.seq_len + t0) * P.head;
        const float *src = (lane ? P.mv[0].v_cache : P.mv[0].k_cache) + (int64_t)layer * P.kv_step + row;
        mbar_arrive_expect_tx(full, kbytes);
        bulk_g2s_plain(pr.ring_base + off + (lane ? voff : 0u), src, kbytes, full);
    } else {
        mbar_arrive(full);   // only the token's own row: nothing travels through the ring
    }
    ++pr.seq;
}

// -------------------------------------------------------------------------------------------------
// consumers
// -------------------------------------------------------------------------------------------------

struct Consumer {
    int seq;             // stages consumed so far (descriptor index = seq mod kFDesc)
    int rb, rround;      // position in the ring of reduction buffers
};

// A lane's sixteen elements of a quantisation group of an input vector: pairs 64 q.. 64 q + 3 from p on, q = 0..3.
__device__ __forceinline__ void issue_pairs(const float2 *p, float4 (&v)[8])
{
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v[2 * q] = ld_pairs2_gpu(p + 64 * q);
        v[2 * q + 1] = ld_pairs2_gpu(p + 64 * q + 2);
    }
}

// Those of them that have not arrived yet are asked for again until they carry `tag`.  While nothing at all has come for
// the warp only an eighth of them is asked for: 148 blocks that poll whole vectors would take as much of the L2 as the
// weight stream does.
__device__ __forceinline__ void poll_pairs(const float2 *p, float4 (&v)[8], int tag, uint32_t sbase, uint64_t wait_ns)
{
    auto all = [&]() {
        bool ok = true;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            ok = ok && tagged(v[q], tag);
        return __all_sync(0xffffffffu, ok) != 0;
    };
    if (all())
        return;
    const long long c0 = sm_clock();
    for (;;) {
        const bool some = tagged(v[0], tag);
        if (!some)
            v[0] = ld_pairs2_gpu(p);
        if (__any_sync(0xffffffffu, some)) {
#pragma unroll
            for (int q = 1; q < 8; ++q)
                if (!tagged(v[q], tag))
                    v[q] = ld_pairs2_gpu(p + 64 * (q >> 1) + 2 * (q & 1));
        }
        if (all())
            return;
        if (__any_sync(0xffffffffu, hand_over_lost(sbase, c0, wait_ns))) {
            set_block_lost(sbase);
            return;
        }
    }
}

// What a thread works on per stage: 32 bytes of each of two rows (16 bytes at two places of the same group) and the two
// groups' headers.
struct StageRegs {
    uint4 w[2][2];
    float2 ms[2];
};

// One matrix-vector phase of the block: prologue (input vector -> fixed-point limbs in shared memory)
// and the block's `nmine` stages.  One copy of this code serves all four phases (the differences are run-time
// parameters): the prologue runs once per phase, so its instructions come from the L2 every time, and four
// inlined copies of it cost more in instruction fetches than the branches cost here.
// in_pairs: the input vector as (value, tag) pairs, or nullptr: plain (p.x_in; the first phase of the launch).
__device__ __forceinline__ void consume_ring_phase(const FusedParams &P, const MvParams &p, int nmine, const float2 *in_pairs, int tag,
                                                   const float *rms_w, uint8_t *smem, uint32_t sbase, Consumer &cs, uint64_t wait_ns,
                                                   int pidx)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int sets = p.rpp >> 1;                  // sets of wpr warps; a set works on two rows of a stage
    const bool active = warp < sets * p.wpr;
    const int rsub = warp / p.wpr;
    const int wi = warp - rsub * p.wpr;
    const int n = p.n;
    uint8_t *share = smem + kFHeader;
    float *scratch = reinterpret_cast<float *>(smem + kFScratch);

    // eight lanes share a quantisation group: lane s of them holds bytes 16 s.. and 128 + 16 s.. of it
    const int g = wi * 4 + (lane >> 3);
    const bool gvalid = active && g < (n >> 8);

    // ---- prologue: the input vector as fixed-point limbs in shared memory.  Every half-warp owns whole quantisation
    // groups of the vector (a lane holds four elements of each quarter of a group) and gives each its own
    // power-of-two scale from the group's largest element: no block-wide maximum has to be agreed on before the
    // conversion can start, and the RMSNorm scalar ss = 1 / sqrt(mean(x^2) + eps) is applied to the dot products
    // at the end (sum_j w_j (r_j ss x_j) = ss sum_j w_j r_j x_j up to rounding), so nothing here waits for the
    // sum of squares either.  Half-warps: 14 warps with a group each would need two rounds for the 16 groups of the 7B shape.
    float *inv_tab = reinterpret_cast<float *>(smem + kFInvTab);   // value of one fixed-point unit, per group
    const int ngroups = n >> 8;
    const bool has_rms = rms_w != nullptr;
    {
        if (tid == 0)
            fused_trace(P, pidx, 0);
        float ssq = 0.f;
#pragma unroll 1
        for (int g0 = 2 * warp; g0 < ngroups; g0 += 2 * kFusedConsWarps) {
            const bool live = g0 + (lane >> 4) < ngroups;          // an odd count of groups: the last half-warp repeats one
            const int gi = live ? g0 + (lane >> 4) : g0;
            const int e = gi * 256 + (lane & 15) * 4;
            float xg[16];
            float4 w4[4];
            if (has_rms) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    w4[q] = ld_cg_f4_issue(rms_w + e + 64 * q);
            }
            if (in_pairs) {
                float4 v[8];
                issue_pairs(in_pairs + e, v);
                poll_pairs(in_pairs + e, v, tag, sbase, wait_ns);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    xg[2 * q] = v[q].x;
                    xg[2 * q + 1] = v[q].z;
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 a4 = ld_cg_f4_issue(p.x_in + e + 64 * q);
                    xg[4 * q] = a4.x; xg[4 * q + 1] = a4.y; xg[4 * q + 2] = a4.z; xg[4 * q + 3] = a4.w;
                }
            }
            if (has_rms) {
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    ssq = fmaf(xg[q], live ? xg[q] : 0.f, ssq);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    xg[4 * q] = __fmul_rn(w4[q].x, xg[4 * q]);
                    xg[4 * q + 1] = __fmul_rn(w4[q].y, xg[4 * q + 1]);
                    xg[4 * q + 2] = __fmul_rn(w4[q].z, xg[4 * q + 2]);
                    xg[4 * q + 3] = __fmul_rn(w4[q].w, xg[4 * q + 3]);
                }
            }
            uint32_t mbits = 0u;
#pragma unroll
            for (int q = 0; q < 16; ++q)
                mbits = max(mbits, __float_as_uint(xg[q]) & 0x7fffffffu);   // non-negative floats order like their bits
            const uint32_t m_lo = __reduce_max_sync(0xffffffffu, lane < 16 ? mbits : 0u);
            const uint32_t m_hi = __reduce_max_sync(0xffffffffu, lane < 16 ? 0u : mbits);
            mbits = lane < 16 ? m_lo : m_hi;
            // 24-bit fixed point: one power-of-two scale per group, |x * f| <= 2^22, so that adding 1.5 * 2^23 leaves the
            // rounded integer in the low bits of the sum (the conversion instruction runs at a quarter of that rate)
            uint32_t z[16];
            int ex = (int)(mbits >> 23) - 126;   // largest < 2^ex for normal numbers
            if (max(m_lo, m_hi) < 0x7e800000u) {           // below 2^126
                if (mbits == 0u)
                    ex = 0;
                ex = max(-90, ex);
                const float f = __int_as_float((127 + 22 - ex) << 23);
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    z[q] = ((uint32_t)__float_as_int(fmaf(xg[q], f, 12582912.0f)) + (0x00008080u - 0x4B400000u)) ^ 0x00008080u;
            } else {                             // infinities, NaN, the very largest: what the conversion instruction makes of them
                float amax = 0.f;
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    amax = fmaxf(amax, fabsf(xg[q]));
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                ex = (int)((__float_as_uint(amax) >> 23) & 0xffu) - 126;
                if (!(amax > 0.f) || !(amax < 3.0e38f))
                    ex = 0;
                ex = max(-90, min(126, ex));
                const float f = __int_as_float((127 + 22 - ex) << 23);
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    z[q] = ((uint32_t)__float2int_rn(xg[q] * f) + 0x00008080u) ^ 0x00008080u;
            }
            if ((lane & 15) == 0)
                inv_tab[gi] = __int_as_float((127 + ex - 22) << 23);
            // three balanced signed byte limbs: after the add-and-flip, bytes 0..2 of z are l0, l1, l2 in
            // [-128, 127] with X = l0 + 256 l1 + 65536 l2
            uint32_t *dst = reinterpret_cast<uint32_t *>(share) + gi * 64 + (lane & 15);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t t0 = __byte_perm(z[4 * q], z[4 * q + 1], 0x5140);
                const uint32_t t2 = __byte_perm(z[4 * q + 2], z[4 * q + 3], 0x5140);
                const uint32_t t1 = __byte_perm(z[4 * q], z[4 * q + 1], 0x0062);
                const uint32_t t3 = __byte_perm(z[4 * q + 2], z[4 * q + 3], 0x0062);
                dst[16 * q] = __byte_perm(t0, t2, 0x5410);
                dst[(n >> 2) + 16 * q] = __byte_perm(t0, t2, 0x7632);
                dst[(n >> 1) + 16 * q] = __byte_perm(t1, t3, 0x5410);
            }
        }
        if (has_rms) {
            ssq = warp_sum(ssq);
            if (lane == 0)
                scratch[warp] = ssq;
        }
    }
    named_barrier_sync(1, kFCons);

    // what a unit of this thread's integer sums is worth: its group's fixed-point unit; the row's sum is multiplied by the
    // RMSNorm scalar when it is complete
    const float unit = gvalid ? inv_tab[g] : 0.f;
    uint32_t xl[2][4][3];
    float xs;
    const uint32_t in_row = (uint32_t)((gvalid ? g * 256 : 0) + (lane & 7) * 16);
    {
        int s0 = 0, s1 = 0, s2 = 0;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const uint4 t = *reinterpret_cast<const uint4 *>(share + (size_t)l * n + in_row + 128 * k);
                xl[k][0][l] = t.x; xl[k][1][l] = t.y; xl[k][2][l] = t.z; xl[k][3][l] = t.w;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                s0 = dp4a_us(0x01010101u, xl[k][q][0], s0);
                s1 = dp4a_us(0x01010101u, xl[k][q][1], s1);
                s2 = dp4a_us(0x01010101u, xl[k][q][2], s2);
            }
        }
        xs = fmaf((float)s2, 65536.0f, fmaf((float)s1, 256.0f, (float)s0));
    }
    float rms = 1.0f;
    if (has_rms) {
        const float ssq = warp_sum(lane < kFusedConsWarps ? scratch[lane] : 0.f);   // the same order in every warp and block
        float tot = __fdiv_rn(ssq, (float)n);
        tot = __fadd_rn(tot, 1e-5f);
        rms = __fdiv_rn(1.0f, __fsqrt_rn(tot));   // RootMeanSquare.java:25-35
    }
    // The limbs, the units and the sums of squares of the next phase take the places of these: a warp may be a whole phase
    // behind another one from here on.
    named_barrier_sync(2, kFCons);
    if (tid == 0)
        fused_trace(P, pidx, 1);

    // Per-thread constants of the stage loop.  The integer pipe runs at half rate and the dot products live on it,
    // so every address computation in the loop costs as much as a dp4a: offsets inside a stage are fixed per
    // thread and phase, shared memory is addressed with 32-bit window addresses, a stage's descriptor is one
    // 16-byte load.  Rows rsub and rsub + sets of a stage (paired: row rsub of either matrix) are this thread's; rows
    // beyond the stage's last are computed from what lies there and not used.
    const int paired = p.paired;
    const uint32_t ring32 = sbase + kFHeader + (uint32_t)P.xarea_bytes;
    const uint32_t row_a = (uint32_t)((active ? rsub : 0) * n) + in_row;
    const uint32_t row_b = row_a + (uint32_t)(sets * n);
    const uint32_t hdr_a = (uint32_t)(p.hdr_off + 8 * ((active ? rsub : 0) * (n >> 8) + (gvalid ? g : 0)));
    const uint32_t hdr_b = hdr_a + (uint32_t)(paired ? p.half_hdr : 8 * sets * (n >> 8));
    const uint32_t desc32 = sbase + kFDescOff;
    uint32_t e = (uint32_t)(cs.seq % kFDesc), parity = (uint32_t)(cs.seq / kFDesc) & 1u;

    auto load = [&](uint32_t at, StageRegs &r) {
        const uint4 d = lds_v4(desc32 + 32u * at);            // off, nrows, e0a, e0b
        const uint32_t slot = ring32 + d.x;
        // rows start on group boundaries: the header of the thread's group is (e0 >> 8) + row * groups per row + g
        r.ms[0] = lds_f2(slot + hdr_a + ((d.z >> 8) << 3));
        r.ms[1] = lds_f2(slot + hdr_b + (((paired ? d.w : d.z) >> 8) << 3));
        r.w[0][0] = lds_v4(slot + row_a);
        r.w[0][1] = lds_v4(slot + row_a + 128u);
        r.w[1][0] = lds_v4(slot + row_b);
        r.w[1][1] = lds_v4(slot + row_b + 128u);
    };

    auto dot = [&](const StageRegs &r, float &va, float &vb) {
        float out[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            int a0 = 0, a1 = 0, a2 = 0;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint4 w = r.w[q][k];
                a0 = dp4a_us(w.x, xl[k][0][0], a0);
                a1 = dp4a_us(w.x, xl[k][0][1], a1);
                a2 = dp4a_us(w.x, xl[k][0][2], a2);
                a0 = dp4a_us(w.y, xl[k][1][0], a0);
                a1 = dp4a_us(w.y, xl[k][1][1], a1);
                a2 = dp4a_us(w.y, xl[k][1][2], a2);
                a0 = dp4a_us(w.z, xl[k][2][0], a0);
                a1 = dp4a_us(w.z, xl[k][2][1], a1);
                a2 = dp4a_us(w.z, xl[k][2][2], a2);
                a0 = dp4a_us(w.w, xl[k][3][0], a0);
                a1 = dp4a_us(w.w, xl[k][3][1], a1);
                a2 = dp4a_us(w.w, xl[k][3][2], a2);
            }
            // |a_l| <= 32 * 255 * 128: the two lower limbs together fit 32 bits
            const float dsum = fmaf((float)a2, 65536.0f, (float)(a1 * 256 + a0));
            out[q] = fmaf(r.ms[q].y, dsum, r.ms[q].x * xs);
        }
        va = out[0];
        vb = out[1];
    };

    auto wait = [&](int t) {
        const uint32_t at = (e + (uint32_t)t) & (kFDesc - 1);
        if (!mbar_wait_bounded(sbase + kFBarFull + 8 * at, parity ^ (at < e ? 1u : 0u), wait_ns))
            set_block_lost(sbase);
        return at;
    };
    auto release = [&](int t) {      // this warp is done with the stage's bytes
        __syncwarp();
        if (lane == 0)
            mbar_arrive(sbase + kFBarEmpty + 8 * ((e + (uint32_t)t) & (kFDesc - 1)));
    };

    // The block's stages are taken in groups of kFGroup: a warp works through a group's rows in one straight line (the
    // bytes of a stage are fetched from shared memory while the dot products of the stage in front run), then folds the
    // partial sums with one butterfly and hands them to the epilogue warp in one go.
    for (int g0 = 0; g0 < nmine; g0 += kFGroup) {
        const int cnt = min(kFGroup, nmine - g0);
        float v[2 * kFGroup];
        if (cnt == kFGroup && active) {
            StageRegs a, b;
            load(wait(0), a);
            if (g0 == 0 && tid == 0)
                fused_trace(P, pidx, 4);
            load(wait(1), b);
            dot(a, v[0], v[1]);
            release(0);
            load(wait(2), a);
            dot(b, v[2], v[3]);
            release(1);
            load(wait(3), b);
            dot(a, v[4], v[5]);
            release(2);
            dot(b, v[6], v[7]);
            release(3);
        } else {
#pragma unroll
            for (int t = 0; t < kFGroup; ++t) {
                v[2 * t] = v[2 * t + 1] = 0.f;
                if (t < cnt) {
                    const uint32_t at = wait(t);
                    if (g0 == 0 && t == 0 && tid == 0)
                        fused_trace(P, pidx, 4);
                    if (active) {
                        StageRegs a;
                        load(at, a);
                        dot(a, v[2 * t], v[2 * t + 1]);
                    }
                    release(t);
                }
            }
        }
        const uint32_t en = (e + (uint32_t)cnt) & (kFDesc - 1);
        parity ^= en < e ? 1u : 0u;
        e = en;
        cs.seq += cnt;
#pragma unroll
        for (int t = 0; t < 2 * kFGroup; ++t)
            v[t] = gvalid ? v[t] * unit : 0.f;
        const float tot = Fold<2 * kFGroup, 16>::run(v, lane) * rms;   // lanes 4 i.. hold the sum of v[i]
        if (cs.rround > 0) {
            if (!mbar_wait_bounded(sbase + kFBarRedEmpty + 8 * cs.rb, (uint32_t)(cs.rround - 1) & 1u, wait_ns))
                set_block_lost(sbase);
        }
        float *red = reinterpret_cast<float *>(smem + kFRedOff + cs.rb * kFRedStride);
        if (active && (lane & 3) == 0) {
            const int t = lane >> 3, r = (lane >> 2) & 1;
            red[(t * p.rpp + r * sets + rsub) * p.wpr + wi] = tot;
        }
        __syncwarp();
        if (lane == 0)
            mbar_arrive(sbase + kFBarRedFull + 8 * cs.rb);
        if (++cs.rb == kFRedBufs) {
            cs.rb = 0;
            ++cs.rround;
        }
    }
    if (tid == 0)
        fused_trace(P, pidx, 2);
}

// The attention step of the block: its run of units, each a stage of cached K and V rows in the ring (the
// token's own row comes straight from the cache in global memory).  One pass with an online softmax per
// lane group; the lane groups of the block are merged through shared memory whenever the head changes.
__device__ __forceinline__ void consume_attention(const FusedParams &P, int tag, const AttSplit &as, uint8_t *smem,
                                                  uint32_t sbase, Consumer &cs, uint64_t wait_ns)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.x;
    const int head = P.head;
    const int u0 = att_first_unit(as, b), u1 = att_first_unit(as, b + 1);
    const int lpp = head >> 2;
    int gw = 1;
    while (gw < lpp)
        gw <<= 1;
    const int ppw = 32 / gw;
    const int g = lane / gw, li = lane - g * gw;
    const bool act = li < lpp;
    const int nslots = kFusedConsWarps * ppw;
    const int slot = warp * ppw + g;
    const int sstride = head + 4;
    float *marea = reinterpret_cast<float *>(smem + kFHeader);
    const float sq = sqrtf((float)head);
    const float2 *kvp = P.kv_pairs;            // the row of this token: keys, then values of all kv heads
    const int kv_dim = P.mv[0].kv_dim;

    // The lane's four elements of up to three vectors of pairs, waited for together; every lane of the warp takes part.
    auto get = [&](const float2 *s0, bool want0, float4 &out0, const float2 *s1, const float2 *s2, bool want12, float4 &out1, float4 &out2) {
        float4 a[6];
#pragma unroll
        for (int z = 0; z < 6; ++z)
            a[z] = make_float4(0.f, 0.f, 0.f, 0.f);
        const long long c0 = sm_clock();
        const int rtag = reader_tag(sbase, tag, L2J_LATE_ROWS);
        for (;;) {
            if (want0) {
                a[0] = ld_pairs2_gpu(s0);
                a[1] = ld_pairs2_gpu(s0 + 2);
            }
            if (want12) {
                a[2] = ld_pairs2_gpu(s1);
                a[3] = ld_pairs2_gpu(s1 + 2);
                a[4] = ld_pairs2_gpu(s2);
                a[5] = ld_pairs2_gpu(s2 + 2);
            }
            const bool ok = (!want0 || (tagged(a[0], rtag) && tagged(a[1], rtag))) &&
                            (!want12 || (tagged(a[2], rtag) && tagged(a[3], rtag) && tagged(a[4], rtag) && tagged(a[5], rtag)));
            if (__all_sync(0xffffffffu, ok))
                break;
            if (__any_sync(0xffffffffu, hand_over_lost(sbase, c0, wait_ns))) {
                set_block_lost(sbase);
                break;
            }
        }
        if (want0)
            out0 = make_float4(a[0].x, a[0].z, a[1].x, a[1].z);
        if (want12) {
            out1 = make_float4(a[2].x, a[2].z, a[3].x, a[3].z);
            out2 = make_float4(a[4].x, a[4].z, a[5].x, a[5].z);
        }
    };
    const int batch_log = __ffs(kAttBatch * ppw) - 1;      // positions per warp and batch: a power of two

    int cur_h = -1, kvh = 0, turn = 0;
    float4 k_own = make_float4(0.f, 0.f, 0.f, 0.f), v_own = k_own;
    static_assert(kAttChunk / kAttBatch <= kFusedConsWarps, "a warp has one batch of a unit at most");
    float4 q4 = make_float4(0.f, 0.f, 0.f, 0.f);
    float m = -INFINITY, l = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);

    float M = -INFINITY, L = 0.f, O = 0.f;   // the block's result for a head: this thread's element of the output
    int others = -1;                         // blocks whose results for the head are merged with this block's
    for (int u = u0;; ++u) {
        const int e = cs.seq % kFDesc;
        FStage d{};
        if (u < u1) {
            if (!mbar_wait_bounded(sbase + kFBarFull + 8 * e, (uint32_t)(cs.seq / kFDesc) & 1u, wait_ns))
                set_block_lost(sbase);
            __syncwarp();     // one descriptor for the whole warp, also behind a wait that ran out in some lanes
            d = *(reinterpret_cast<const FStage *>(smem + kFDescOff) + e);
        }
        const int h = u < u1 ? d.seg : -1;
        const bool fresh = h != cur_h;
        if (fresh) {
            if (cur_h >= 0) {
                // merge the lane groups in slot order and write the block's partial of head h
                float *mine = marea + slot * sstride;
                if (act)
                    *reinterpret_cast<float4 *>(mine + 4 * li) = acc;
                if (li == 0) {
                    mine[head] = m;
                    mine[head + 1] = l;
                }
                named_barrier_sync(2, kFCons);
                if (tid < ((head + 31) & ~31)) {
                    // the weights of 32 slots at a time, one per lane and once per warp; then every thread its element
                    float O2 = 0.f;
                    M = -INFINITY;
                    L = O = 0.f;
                    for (int s = lane; s < nslots; s += 32)
                        M = fmaxf(M, marea[s * sstride + head]);
                    M = warp_max(M);
                    const float *col = marea + (tid < head ? tid : 0);
                    for (int s0 = 0; s0 < nslots; s0 += 32) {
                        const int s1 = min(32, nslots - s0);
                        float w = 0.f;
                        if (lane < s1) {
                            const float2 ml = *reinterpret_cast<const float2 *>(marea + (s0 + lane) * sstride + head);
                            if (ml.y > 0.f)
                                w = expf(ml.x - M);
                            L = fmaf(ml.y, w, L);
                        }
                        for (int s = 0; s < s1; s += 2) {
                            O = fmaf(col[(s0 + s) * sstride], __shfl_sync(0xffffffffu, w, s), O);
                            if (s + 1 < s1)
                                O2 = fmaf(col[(s0 + s + 1) * sstride], __shfl_sync(0xffffffffu, w, s + 1), O2);
                        }
                    }
                    L = warp_sum(L);
                    O += O2;
                    const int pslot = b - att_block_of(as, cur_h * as.nchunk);
                    others = pslot == 0 ? att_partials(as, cur_h) - 1 : -1;
                    if (pslot > 0) {
                        float2 *out = P.att_pairs + ((int64_t)cur_h * (kAttSlots - 1) + pslot - 1) * (head + 2);
                        if (tid < head)
                            st_pair_gpu(out + tid, O, tag);
                        if (tid == 0) {
                            st_pair_gpu(out + head, M, tag);
                            st_pair_gpu(out + head + 1, L, tag);
                        }
                    } else if (others == 0 && tid < head) {
                        // ExpSumNormalize.java:33-37 folded into the weighted sum
                        st_pair_gpu(P.o_pairs + (int64_t)cur_h * head + tid, __fdiv_rn(O, L), tag);
                    }
                }
                named_barrier_sync(2, kFCons);   // the merge area is free again
            }
            if (u == u1)
                break;
            cur_h = h;
            m = -INFINITY;
            l = 0.f;
            acc = make_float4(0.f, 0.f, 0.f, 0.f);
            kvh = h / P.kv_mul;
        }
        // the row that this token's QKV phase has just written is the unit's last one, if it is in it at all
        const bool has_own = d.nrows > d.e0a;
        if (fresh || has_own)
            get(P.q_pairs + (int64_t)h * head + 4 * li, fresh && act, q4, kvp + (int64_t)kvh * head + 4 * li,
                kvp + kv_dim + (int64_t)kvh * head + 4 * li, has_own && act, k_own, v_own);
        const float *ks = reinterpret_cast<const float *>(smem + kFHeader + P.xarea_bytes + (size_t)d.off);
        const float *vs = reinterpret_cast<const float *>(smem + kFHeader + P.xarea_bytes + (size_t)d.off + (size_t)d.aux);
        // A lane group takes kAttBatch positions at a time (independent chains of dot products and shuffles).  A unit is too
        // small for all warps: the next one starts with the warp behind the last one that had work.
        const int batches = (d.nrows + (1 << batch_log) - 1) >> batch_log;      // at most kAttChunk / kAttBatch = 8
        int mine = warp - turn;
        mine += mine < 0 ? kFusedConsWarps : 0;
        turn += batches;
        turn -= turn >= kFusedConsWarps ? kFusedConsWarps : 0;
        if (mine < batches) {
            const int first = (mine * ppw + g) * kAttBatch;
            float4 kk[kAttBatch], vv[kAttBatch];
#pragma unroll
            for (int t = 0; t < kAttBatch; ++t) {
                kk[t] = vv[t] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (act && first + t < d.e0a) {
                    kk[t] = *reinterpret_cast<const float4 *>(ks + (size_t)(first + t) * head + 4 * li);
                    vv[t] = *reinterpret_cast<const float4 *>(vs + (size_t)(first + t) * head + 4 * li);
                }
            }
            if (has_own) {
#pragma unroll
                for (int t = 0; t < kAttBatch; ++t)
                    if (first + t == d.e0a) {
                        kk[t] = k_own;
                        vv[t] = v_own;
                    }
            }
            float s[kAttBatch];
#pragma unroll
            for (int t = 0; t < kAttBatch; ++t) {
                float dd = kk[t].x * q4.x;
                dd = fmaf(kk[t].y, q4.y, dd);
                dd = fmaf(kk[t].z, q4.z, dd);
                s[t] = fmaf(kk[t].w, q4.w, dd);
            }
            for (int o = gw >> 1; o > 0; o >>= 1) {
#pragma unroll
                for (int t = 0; t < kAttBatch; ++t)
                    s[t] += __shfl_xor_sync(0xffffffffu, s[t], o);
            }
            float mloc = -INFINITY;
#pragma unroll
            for (int t = 0; t < kAttBatch; ++t) {
                s[t] = first + t < d.nrows ? __fdiv_rn(s[t], sq) : -INFINITY;   // AttentionLoop.java:48
                mloc = fmaxf(mloc, s[t]);
            }
            if (mloc > -INFINITY) {
                const float mn = fmaxf(m, mloc);
                const float sc = expf(m - mn);
                l *= sc;
                acc.x *= sc; acc.y *= sc; acc.z *= sc; acc.w *= sc;
#pragma unroll
                for (int t = 0; t < kAttBatch; ++t) {
                    const float pw = expf(s[t] - mn);
                    l += pw;
                    acc.x = fmaf(pw, vv[t].x, acc.x);
                    acc.y = fmaf(pw, vv[t].y, acc.y);
                    acc.z = fmaf(pw, vv[t].z, acc.z);
                    acc.w = fmaf(pw, vv[t].w, acc.w);
                }
                m = mn;
            }
        }
        __syncwarp();
        if (lane == 0)
            mbar_arrive(sbase + kFBarEmpty + 8 * e);
        ++cs.seq;
    }
    // The block with a head's first positions merges the partial results of the others (the blocks behind it, in block
    // order) and hands the finished output on.  A head that others work on too is the block's last one, so nobody waits for a
    // block that waits.
    if (others > 0 && tid < ((head + 31) & ~31)) {
        const float2 *parts = P.att_pairs + (int64_t)cur_h * (kAttSlots - 1) * (head + 2);
        const float2 *src = parts + (tid < head ? tid : 0);
        const float2 *src_ml = parts + (int64_t)min(lane, others - 1) * (head + 2) + head;   // lane z: maximum and sum of partial z
        float2 o[kAttSlots - 1];
        float4 ml = ld_pairs2_gpu(src_ml);
#pragma unroll
        for (int z = 0; z < kAttSlots - 1; ++z)
            if (z < others)
                o[z] = ld_pair_gpu(src + (int64_t)z * (head + 2));
        const long long c0 = sm_clock();
        const int ptag = reader_tag(sbase, tag, L2J_LATE_PARTIALS);
        for (;;) {
            bool ok = tagged(ml, ptag);
#pragma unroll
            for (int z = 0; z < kAttSlots - 1; ++z)
                if (z < others)
                    ok = ok && __float_as_int(o[z].y) == ptag;
            if (__all_sync(0xffffffffu, ok))
                break;
            if (__any_sync(0xffffffffu, hand_over_lost(sbase, c0, wait_ns))) {
                set_block_lost(sbase);
                break;
            }
            if (!tagged(ml, ptag))
                ml = ld_pairs2_gpu(src_ml);
#pragma unroll
            for (int z = 0; z < kAttSlots - 1; ++z)
                if (z < others && __float_as_int(o[z].y) != ptag)
                    o[z] = ld_pair_gpu(src + (int64_t)z * (head + 2));
        }
        const float gm = fmaxf(M, warp_max(ml.x));
        const float w0 = L > 0.f ? expf(M - gm) : 0.f;
        const float w = lane < others && ml.z > 0.f ? expf(ml.x - gm) : 0.f;
        L = fmaf(L, w0, warp_sum(ml.z * w));
        O *= w0;
#pragma unroll
        for (int z = 0; z < kAttSlots - 1; ++z) {
            const float wz = __shfl_sync(0xffffffffu, w, z);
            if (z < others)
                O = fmaf(o[z].x, wz, O);
        }
        if (tid < head)
            st_pair_gpu(P.o_pairs + (int64_t)cur_h * head + tid, __fdiv_rn(O, L), tag);
    }
}

// -------------------------------------------------------------------------------------------------
// epilogue warp
// -------------------------------------------------------------------------------------------------

struct Epilogue {
    int rb, rround;
};

// Results leave as (value, tag) pairs, one store each, which the readers poll: no fence, no counter and no second trip to the
// L2.  resid: where the old value of a residual element comes from (pairs of `resid_tag`, or the plain vector p.y before the
// first one).  plain: the last layer, whose query, hidden vector and residual stream stay readable behind the launch.
__device__ __forceinline__ void epilogue_phase(const FusedParams &P, const MvParams &p, int layer, int first, int nmine, int pos,
                                               uint8_t *smem, uint32_t sbase, Epilogue &es, uint64_t wait_ns, float2 *out, int tag,
                                               const float2 *resid, int resid_tag, bool plain)
{
    const int lane = threadIdx.x & 31;
    const int G = gridDim.x;
    const int sets = p.rpp >> 1;
    const int wpr = p.wpr;
    const int rs = p.rs;                 // output rows (row pairs) per stage
    const float *rope_c = reinterpret_cast<const float *>(smem + kFRopeOff);
    const float *rope_s = rope_c + 64;
    const int per = p.epilogue == EPI_QKV_ROPE ? rs >> 1 : rs;   // results (rotated pairs of rows) of a stage
    for (int g0 = 0; g0 < nmine; g0 += kFGroup) {
        const int cnt = min(kFGroup, nmine - g0);
        const float *red = reinterpret_cast<const float *>(smem + kFRedOff + es.rb * kFRedStride);
        for (int i0 = 0; i0 < cnt * per; i0 += 32) {
            const int idx = i0 + lane;
            const int t = idx / per, i = idx - t * per;
            int seg = 0, row0 = 0, nrows = 0;
            if (t < cnt)
                stage_rows(p, first + (g0 + t) * G, seg, row0, nrows);
            const int ri = p.epilogue == EPI_QKV_ROPE ? 2 * i : i;
            const bool mine = t < cnt && ri < nrows;
            const int row = row0 + ri;
            float2 old = make_float2(0.f, 0.f);
            if (p.epilogue == EPI_RESIDUAL && mine) {   // ahead of the sums
                if (resid)
                    old = ld_pair_gpu(resid + row);
                else
                    old.x = __ldcg(p.y + row);
            }
            // everything that does not need the sums is done ahead of them too
            int kvh = 0, d = 0;
            float c = 1.f, sn = 0.f;
            if (p.epilogue == EPI_QKV_ROPE && mine) {
                kvh = row / p.head;
                d = row - kvh * p.head;
                if (seg != 2) {
                    c = rope_c[d >> 1];
                    sn = rope_s[d >> 1];
                }
            }
            if (i0 == 0) {
                if (!mbar_wait_bounded(sbase + kFBarRedFull + 8 * es.rb, (uint32_t)es.rround & 1u, wait_ns))
                    set_block_lost(sbase);
            }
            if (!mine)
                continue;
            const float *ra = red + (t * p.rpp + ri) * wpr;
            const float *rb = p.epilogue == EPI_SWIGLU ? ra + sets * wpr : ra + wpr;    // partner row: of W3, or the next one
            const bool two = p.epilogue != EPI_RESIDUAL;
            float v0 = 0.f, v1 = 0.f;
#pragma unroll 4
            for (int w = 0; w < wpr; ++w) {
                v0 += ra[w];
                if (two)
                    v1 += rb[w];
            }
            if (p.epilogue == EPI_QKV_ROPE) {
                // a lane owns a pair of rows: (v0, v1) are rotated together (ApplyRope.java:61-92)
                float r0 = v0, r1 = v1;
                if (seg != 2) {
                    r0 = __fsub_rn(__fmul_rn(v0, c), __fmul_rn(v1, sn));
                    r1 = __fadd_rn(__fmul_rn(v0, sn), __fmul_rn(v1, c));
                }
                float2 *dst = seg == 0 ? out + row : P.kv_pairs + (seg == 2 ? p.kv_dim : 0) + row;
                st_pair_gpu(dst, r0, tag);
                st_pair_gpu(dst + 1, r1, tag);
                if (seg == 0 && plain) {
                    p.q_out[row] = r0;
                    p.q_out[row + 1] = r1;
                }
                if (seg != 0) {      // the cache is for the tokens behind this one
                    float *cache = (seg == 2 ? p.v_cache : p.k_cache) + (int64_t)layer * P.kv_step + ((int64_t)kvh * p.seq_len + pos) * p.head + d;
                    cache[0] = r0;
                    cache[1] = r1;
                }
            } else if (p.epilogue == EPI_SWIGLU) {
                const float r = __fmul_rn(__fmul_rn(v0, sigmoid_accurate(v0)), v1);   // Silu.java:122-132 order
                st_pair_gpu(out + row, r, tag);
                if (plain)
                    p.y[row] = r;
            } else {   // EPI_RESIDUAL
                if (resid && __float_as_int(old.y) != resid_tag) {
                    const long long c0 = sm_clock();
                    do {
                        old = ld_pair_gpu(resid + row);
                        if (hand_over_lost(sbase, c0, wait_ns)) {
                            set_block_lost(sbase);
                            break;
                        }
                    } while (__float_as_int(old.y) != resid_tag);
                }
                const float r = __fadd_rn(old.x, v0);
                st_pair_gpu(out + row, r, tag);
                if (plain && resid == P.xa_pairs)
                    p.y[row] = r;
            }
        }
        __syncwarp();
        if (lane == 0)
            mbar_arrive(sbase + kFBarRedEmpty + 8 * es.rb);
        if (++es.rb == kFRedBufs) {
            es.rb = 0;
            ++es.rround;
        }
    }
}

}  // namespace

// =============================================================================================
// the kernel
// =============================================================================================

__global__ void __launch_bounds__(kFusedThreads, 1) fused_layers_kernel(const __grid_constant__ FusedParams P)
{
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.x, G = gridDim.x;
    const uint32_t sbase = smem_u32(smem);
    const uint64_t wait_ns = (uint64_t)P.timeout_us * 1000ull;

    if (tid < kFDesc) {
        mbar_init(sbase + kFBarFull + 8 * tid, 4);         // the four producer lanes
        mbar_init(sbase + kFBarEmpty + 8 * tid, kFusedConsWarps);
    }
    if (tid < kFRedBufs) {
        mbar_init(sbase + kFBarRedFull + 8 * tid, kFusedConsWarps);
        mbar_init(sbase + kFBarRedEmpty + 8 * tid, 1);
    }
    if (tid == 0)
        *reinterpret_cast<volatile int *>(smem + kFLost) = 0;
    if (tid < 32)
        mbar_fence_init();
    __syncthreads();
    pdl_launch_dependents();   // the classifier kernel behind may take the SMs as they free up

    // ------------------------------------------------------------------------------ producer
    if (warp == kFusedConsWarps) {
        if (lane >= 4)
            return;
        Producer pr;
        pr.smem = smem;
        pr.sbase = sbase;
        pr.ring_base = sbase + kFHeader + (uint32_t)P.xarea_bytes;
        pr.vhead = 0;
        pr.ring_bytes = P.ring_bytes;
        pr.seq = pr.tail = pr.vtail = 0;
        pr.wait_ns = wait_ns;
        const uint64_t pol = policy_evict_first();
        pr.pos = -1;
        pr.as = AttSplit{};
        pr.off = 0;
        int rot = 0;
        for (int layer = 0; layer < P.n_layers; ++layer) {
            if (pr.vhead > kFRebase)
                pr.rebase(lane);
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                const MvParams &p = P.mv[k];
                const int S = p.total_stages;
                if (!(P.debug_no_copy & 8) && lane == 0) fused_trace(P, layer * 5 + (k == 0 ? 0 : k + 1), 5);
                produce_phase(pr, P, p, k, layer, first_stage_of(b, rot, G), G, pol, lane);
                if (!(P.debug_no_copy & 8) && lane == 0) fused_trace(P, layer * 5 + (k == 0 ? 0 : k + 1), 6);
                rot = (rot + S) % G;
                if (k == 0) {
                    producer_learn_pos(pr, P, G);
                    if (b < pr.as.ga) {
                        const int u0 = att_first_unit(pr.as, b), u1 = att_first_unit(pr.as, b + 1);
                        if (lane == 0) fused_trace(P, layer * 5 + 1, 5);
                        for (int u = u0; u < u1; ++u) {
                            if (pr.vhead > kFRebase)
                                pr.rebase(lane);
                            produce_att_stage(pr, P, layer, u, pr.as, pr.pos, lane);
                        }
                        if (lane == 0) fused_trace(P, layer * 5 + 1, 6);
                    }
                }
            }
        }
        // No copy of this block may still be in flight when its shared memory is handed to the next block: the
        // consumers have waited for every stage, so these waits return at once unless a wait ran out before.
        for (int d = max(pr.tail, pr.seq - kFDesc); d < pr.seq; ++d)
            mbar_wait_bounded(sbase + kFBarFull + 8 * (d % kFDesc), (uint32_t)(d / kFDesc) & 1u, wait_ns);
        __syncwarp(0xfu);
        if (lane == 0 && block_lost(sbase))
            atomicOr(&P.state->status, L2J_DS_WAIT_TIMEOUT);
        return;
    }

    // Everything below reads what the kernel in front wrote (x, the position).
    pdl_wait();
    const int pos = __ldcg(&P.state->cur_pos);
    const AttSplit as = att_split(P, pos, G);
    const unsigned int epoch = __ldcg(P.epoch);
    const int tag0 = (int)(epoch * (unsigned int)P.n_layers) + 1;    // tag of layer l: tag0 + l
    *reinterpret_cast<volatile int *>(smem + kFLate) = (int)__ldcg(P.epoch + 1);    // the same from every thread
    if ((__ldcg(&P.state->status) & L2J_DS_WAIT_TIMEOUT) != 0)
        set_block_lost(sbase);

    // ------------------------------------------------------------------------------ epilogue warp
    if (warp == kFusedConsWarps + 1) {
        Epilogue es;
        es.rb = es.rround = 0;
        // Every forward before this one has bumped the last phase's counter once per block.  If one is missing, the blocks of the
        // context (or its host) have lost count: reported here too, because a stage of a layer split has no classifier that waits.
        if (b == 0 && lane == 0 && ld_acquire_u32(P.sync + (int64_t)kSyncStride * (5 * P.n_layers - 1)) != (epoch - 1u) * (unsigned int)G)
            atomicOr(&P.state->status, L2J_DS_WAIT_TIMEOUT);
        {
            float *rope_c = reinterpret_cast<float *>(smem + kFRopeOff);
            const int half = P.head >> 1;
            for (int i = lane; i < half; i += 32) {
                rope_c[i] = __ldg(P.mv[0].rope_cos + (int64_t)pos * half + i);
                rope_c[64 + i] = __ldg(P.mv[0].rope_sin + (int64_t)pos * half + i);
            }
            __syncwarp();
        }
        int rot = 0;
        for (int layer = 0; layer < P.n_layers; ++layer) {
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                const MvParams &p = P.mv[k];
                const int S = p.total_stages;
                const int first = first_stage_of(b, rot, G);
                const int nmine = first < S ? (S - first + G - 1) / G : 0;
                rot = (rot + S) % G;
                const int tag = tag0 + layer;
                float2 *out = k == 0 ? P.q_pairs : (k == 1 ? P.xa_pairs : (k == 2 ? P.h_pairs : P.xb_pairs));
                const float2 *resid = k == 1 ? (layer > 0 ? P.xb_pairs : nullptr) : P.xa_pairs;
                const bool last = layer + 1 == P.n_layers;
                int rtag = k == 1 ? tag - 1 : tag;
                if (k == 3 && last && lane > 0)
                    rtag = reader_tag(sbase, rtag, L2J_LATE_RESIDUAL);
                epilogue_phase(P, p, layer, first, nmine, pos, smem, sbase, es, wait_ns, out, tag, resid, rtag, last);
                if (k == 3 && last) {
                    // the classifier kernel behind polls this counter: every result of the block in this phase was written by
                    // this warp, the release is cumulative
                    __syncwarp();
                    if (lane == 0)
                        red_release_add_u32(P.sync + (int64_t)kSyncStride * (layer * 5 + 4), 1u);
                }
                if (lane == 0)
                    fused_trace(P, layer * 5 + (k == 0 ? 0 : k + 1), 3);
            }
        }
        __syncwarp();
        if (lane == 0 && block_lost(sbase))
            atomicOr(&P.state->status, L2J_DS_WAIT_TIMEOUT);
        return;
    }

    // ------------------------------------------------------------------------------ consumers
    Consumer cs;
    cs.seq = 0;
    cs.rb = cs.rround = 0;
    int rot = 0;
    for (int layer = 0; layer < P.n_layers; ++layer) {
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            const MvParams &p = P.mv[k];
            const int S = p.total_stages;
            const int first = first_stage_of(b, rot, G);
            const int nmine = first < S ? (S - first + G - 1) / G : 0;
            rot = (rot + S) % G;
            const int pidx = layer * 5 + (k == 0 ? 0 : k + 1);
            if (nmine > 0) {
                if (tid == 0)
                    fused_trace(P, pidx, 7);
                const float *rms_w = p.rms_w ? p.rms_w + (int64_t)layer * P.rms_step : nullptr;
                // the first phase's input came from the kernel in front
                const float2 *in = k == 0 ? (layer > 0 ? P.xb_pairs : nullptr) : (k == 1 ? P.o_pairs : (k == 2 ? P.xa_pairs : P.h_pairs));
                const int tag = k == 0 ? tag0 + layer - 1 : tag0 + layer;
                consume_ring_phase(P, p, nmine, in, reader_tag(sbase, tag, L2J_LATE_INPUT), rms_w, smem, sbase, cs, wait_ns, pidx);
            }
            if (k == 0) {
                // attention over positions 0..pos (Run.java:450-478)
                const int aidx = layer * 5 + 1;
                if (b < as.ga) {
                    if (tid == 0)
                        fused_trace(P, aidx, 0);
                    consume_attention(P, tag0 + layer, as, smem, sbase, cs, wait_ns);
                    if (tid == 0)
                        fused_trace(P, aidx, 2);
                    if (tid == 0)
                        fused_trace(P, aidx, 3);
                }
            }
        }
    }
    __syncwarp();
    if (lane == 0 && block_lost(sbase))
        atomicOr(&P.state->status, L2J_DS_WAIT_TIMEOUT);
}

// max_smem: shared memory that a block may have; resident: how many blocks of want_smem bytes (max_smem at most) the device holds at once.
cudaError_t prepare_fused(int want_smem, int *max_smem, int *resident)
{
    int dev = 0, optin = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess)
        return e;
    *max_smem = optin;
    if ((e = cudaFuncSetAttribute(fused_layers_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin)) != cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(fused_layers_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared)) != cudaSuccess)
        return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fused_layers_kernel, kFusedThreads,
                                                      (size_t)(want_smem < optin ? want_smem : optin));
    *resident = per_sm * sms;
    return e;
}

cudaError_t launch_fused(cudaStream_t stream, bool pdl, int grid, int smem_bytes, const FusedParams &p)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kFusedThreads);
    cfg.dynamicSmemBytes = (size_t)smem_bytes;
    cfg.stream = stream;
    // Cooperative: the blocks wait for each other, so either all of them get onto the device or none does, also while another
    // context's persistent kernel wants the same SMs.  Costs nothing that can be measured (4 layers of dim 1280, 400 forwards: 39.5 ms
    // with and without).
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, fused_layers_kernel, p);
}

}  // namespace l2j
