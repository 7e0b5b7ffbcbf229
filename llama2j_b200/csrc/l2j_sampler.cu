// Temperature / top-p token selection on the device, reproducing the reference's host-side Sampler bit for
// bit, so that `--temp 0.9 --seed S` chooses the tokens the Java program would choose from the same logits
// and only the chosen id (4 bytes) crosses PCIe instead of the 128 KB of logits.
//
// Reference (paths relative to src/main/java/com/lastbot/llama2j/):
//   Run.java:643-665        logits /= temperature; FindMax.call; ExpSumNormalize.call (exp in double, the sum
//                           one sequential float accumulator); Sampler.sample or Sampler.sample_topp
//   Sampler.java:20-44      java.util.Random.nextFloat() (48-bit LCG), the cumulative walk
//   Sampler.java:76-120     top-p: candidates >= (1 - topp) / (n - 1) in index order into the FIRST n0 entries of
//                           a ProbIndex array that lives as long as the Sampler, a STABLE descending sort of the
//                           WHOLE array (so entries that earlier calls left beyond n0 take part), the
//                           cumulative cut, the draw
//
// One cluster of eight blocks, which reach each other's shared memory.  What bounds it is a chain of dependent
// steps, not bytes (the whole state is under 1 MB).  One forward and one choice at the 110M shape (vocabulary 32000,
// temperature 0.9, top-p 0.9) take 380 us, of which the forward is 290; with one block, the sums by one thread and an
// eight-pass sort of the whole array they took 1645 us.
//
//   sums     The softmax sum and the cumulative sums have to be the reference's sequential float sums.  While the
//            running sum stays inside one binade its ulp is fixed, and adding an element moves the sum by a whole
//            number of ulps that depends on the element and, where it is exactly half way, on the parity of the
//            sum.  Such steps compose associatively (a pair of increments, one per parity), so a window of 4096
//            elements is one block-wide scan; the element at which the sum leaves the binade is found, added with
//            an ordinary float addition, and the next window starts behind it.  Bit for bit the sequential sum.
//   sort     Only the n0 candidates are new; what stands behind them in the array is the tail of the previous
//            call's sorted array and still sorted (all zeros at first).  So the candidates alone are sorted (each
//            block its share, a stable radix sort in shared memory) and every element's place in the stable sort of
//            the whole array is its place in its own list plus its counts in the other lists (binary searches).

#include "l2j_device.cuh"
#include "l2j_internal.h"

#include <cooperative_groups.h>

#include <cfloat>
#include <cmath>

namespace l2j {

namespace {

namespace cg = cooperative_groups;

constexpr int kSampThreads = 1024, kSampWarps = kSampThreads / 32;
constexpr int kSampCtas = 8;                       // blocks of the cluster (the portable maximum)
constexpr int kSampRows = 5;                       // elements per thread of a block's share of the vocabulary
constexpr int kSampMaxVocab = 39936;               // what the entry point takes
static_assert(kSampMaxVocab <= kSampCtas * kSampRows * kSampThreads, "every element has a thread");
constexpr int kDigitBits = 8, kDigits = 1 << kDigitBits;
constexpr int kHistBytes = kDigits * kSampWarps * 2;
constexpr int kSegRows = kSampRows;                // rows of 32 elements per warp in the local sort
constexpr int kFirstSerial = 256;                  // elements added by one thread before the first window

__device__ __forceinline__ int rng_next(unsigned long long &rng, int bits)
{
    rng = (rng * 0x5DEECE66DULL + 0xBULL) & ((1ULL << 48) - 1ULL);
    return (int)((long long)rng >> (48 - bits));
}

__device__ __forceinline__ float rng_next_float(unsigned long long &rng)
{
    return __fdiv_rn((float)rng_next(rng, 24), 16777216.0f);
}

// ---- the reference's sequential float sum, scanned

// How a run of elements moves the running sum, in ulps of its binade: by `e` if the sum is even, by `o` if it is odd.
// Saturated: past 2^24 the sum has left the binade and only that fact counts.
struct Step {
    int e, o;
};

constexpr int kStepMax = 1 << 26;

__device__ __forceinline__ Step step_then(const Step &f, const Step &g)
{
    Step h;
    h.e = min(f.e + ((f.e & 1) ? g.o : g.e), kStepMax);
    h.o = min(f.o + ((f.o & 1) ? g.e : g.o), kStepMax);
    return h;
}

// x: the element in ulps (exact: a power of two times the element).  A NaN leaves the binade too: the element is then
// added with an ordinary addition.
__device__ __forceinline__ Step step_of(float x)
{
    if (!(x < 33554432.0f))
        return Step{1 << 25, 1 << 25};
    const int a = (int)x;
    const float f = x - (float)a;
    if (f == 0.5f)   // half way: to the even neighbour
        return Step{a + (a & 1), a + 1 - (a & 1)};
    const int r = a + (f > 0.5f ? 1 : 0);
    return Step{r, r};
}

struct ScanShared {
    Step warp[kSampWarps];
    int first;       // first thread of the window that stops it
    float sum;       // the sum behind that thread's elements (or behind the window)
    int hit;         // element at which the sum exceeded the threshold, or -1
};

// The first of the four sums behind elements i .. i + 3 that exceeds the limit (-1: none), and that sum (else the last).
// A later element that is NaN does not hide an earlier sum.
__device__ __forceinline__ int first_above(const float4 &c, int i, float limit, float &sum)
{
    sum = c.x > limit ? c.x : (c.y > limit ? c.y : (c.z > limit ? c.z : c.w));
    return c.x > limit ? i : (c.y > limit ? i + 1 : (c.z > limit ? i + 2 : (c.w > limit ? i + 3 : -1)));
}

// Adds v[0 .. n) in order to `sum` (block-wide; v in shared memory, 16-byte aligned, readable up to the next multiple
// of four) and returns the first i with (sum after element i) > limit, or -1; `sum` becomes the sum behind that element
// or behind all of them.  keep: the running sums replace the elements (up to the stop).  A sum that is NaN stays NaN and
// exceeds nothing, so it ends the walk (nobody asks for the running sums then).
__device__ int sequential_sum(float *v, int n, float &sum, float limit, bool keep, ScanShared &sh)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int i0 = 0, serial = kFirstSerial;
    while (i0 < n) {
        if (sum != sum)
            return -1;
        if (i0 < serial || !(sum >= 1e-30f && sum < INFINITY)) {
            // the first elements (many binades in few steps), sums so small that an element in ulps could overflow, infinity
            const int end = min(n, i0 + kFirstSerial);
            if (tid == 0) {
                float s = sum;
                int hit = -1;
                for (int i = i0; i < end && hit < 0; i += 4) {
                    float4 x = *reinterpret_cast<const float4 *>(v + i);
                    x.x = __fadd_rn(s, x.x);
                    x.y = i + 1 < n ? __fadd_rn(x.x, x.y) : x.x;
                    x.z = i + 2 < n ? __fadd_rn(x.y, x.z) : x.y;
                    x.w = i + 3 < n ? __fadd_rn(x.z, x.w) : x.z;
                    s = x.w;
                    if (keep)
                        *reinterpret_cast<float4 *>(v + i) = x;
                    if (!(s <= limit))
                        hit = first_above(x, i, limit, s);
                }
                sh.sum = s;
                sh.hit = hit;
            }
            __syncthreads();
            sum = sh.sum;
            const int hit = sh.hit;
            __syncthreads();
            if (hit >= 0)
                return hit;
            i0 = end;
            serial = 0;
            continue;
        }
        const int ex = (int)((__float_as_uint(sum) >> 23) & 0xffu) - 127;      // sum is normal: in [2^ex, 2^(ex + 1))
        const float to_ulps = __int_as_float((127 + 23 - ex) << 23);
        const int s0 = (int)(__float_as_uint(sum) & 0x7fffffu) | 0x800000;     // sum in ulps
        const int i = i0 + 4 * tid;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n) {
            x = *reinterpret_cast<const float4 *>(v + i);
            if (i + 1 >= n) x.y = 0.f;
            if (i + 2 >= n) x.z = 0.f;
            if (i + 3 >= n) x.w = 0.f;
        }
        Step st = step_then(step_then(step_of(x.x * to_ulps), step_of(x.y * to_ulps)),
                            step_then(step_of(x.z * to_ulps), step_of(x.w * to_ulps)));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            Step before;
            before.e = __shfl_up_sync(0xffffffffu, st.e, o);
            before.o = __shfl_up_sync(0xffffffffu, st.o, o);
            if (lane >= o)
                st = step_then(before, st);
        }
        if (lane == 31)
            sh.warp[warp] = st;
        if (tid == 0)
            sh.first = kSampThreads;
        __syncthreads();
        Step ws = sh.warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            Step before;
            before.e = __shfl_up_sync(0xffffffffu, ws.e, o);
            before.o = __shfl_up_sync(0xffffffffu, ws.o, o);
            if (lane >= o)
                ws = step_then(before, ws);
        }
        // the steps of the warps in front, then of the lanes in front
        const int pw = max(warp - 1, 0), pl = max(lane - 1, 0);
        Step fw, fl;
        fw.e = __shfl_sync(0xffffffffu, ws.e, pw);
        fw.o = __shfl_sync(0xffffffffu, ws.o, pw);
        fl.e = __shfl_sync(0xffffffffu, st.e, pl);
        fl.o = __shfl_sync(0xffffffffu, st.o, pl);
        if (warp == 0)
            fw = Step{0, 0};
        if (lane == 0)
            fl = Step{0, 0};
        int at = s0 + ((s0 & 1) ? fw.o : fw.e);
        const int end_w = at + ((at & 1) ? st.o : st.e);
        at += (at & 1) ? fl.o : fl.e;
        const bool live = at < (1 << 24);                  // the sum has not left the binade in front of this thread
        float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
        bool stop = false;
        if (live) {
            c.x = __fadd_rn((float)at * __int_as_float((127 - 23 + ex) << 23), x.x);   // the sum in front, exact
            c.y = __fadd_rn(c.x, x.y);
            c.z = __fadd_rn(c.y, x.z);
            c.w = __fadd_rn(c.z, x.w);
            stop = end_w >= (1 << 24) || c.w > limit;
            if (keep && i < n)
                *reinterpret_cast<float4 *>(v + i) = c;
            if (stop)
                atomicMin(&sh.first, tid);
        }
        __syncthreads();
        const int first = sh.first;
        if (tid == min(first, kSampThreads - 1)) {
            float s;
            sh.hit = first_above(c, i, limit, s);
            sh.sum = s;
        }
        __syncthreads();
        sum = sh.sum;
        if (sh.hit >= 0)
            return sh.hit;
        i0 += 4 * (min(first, kSampThreads - 1) + 1);
    }
    return -1;
}

// ---- stable descending sort of a block's candidates in shared memory

// Exclusive prefix sum of one value per thread over the block.
__device__ __forceinline__ int block_exclusive_scan(int v, int *warp_sums, int &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o)
            inc += t;
    }
    if (lane == 31)
        warp_sums[warp] = inc;
    __syncthreads();
    int w = warp_sums[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o)
            w += t;
    }
    total = __shfl_sync(0xffffffffu, w, 31);
    const int base = warp > 0 ? __shfl_sync(0xffffffffu, w, max(warp - 1, 0)) : 0;
    __syncthreads();
    return base + inc - v;
}

// Least-significant-digit radix sort on ~bits (non-negative floats order like their bits), four passes between
// (k0, i0) and (k1, i1); the result is in (k0, i0).  A warp owns a contiguous run of rows of 32 elements, so that
// counting per (digit, warp) in warp order and ranking inside a row by lane keeps equal keys in order.
__device__ void sort_local(float *k0, int *i0, float *k1, int *i1, int m, unsigned short *hist, int *warp_sums)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rows = (m + 32 * kSampWarps - 1) / (32 * kSampWarps);   // rows per warp, at most kSegRows
    const int base = warp * rows * 32 + lane;
    for (int pass = 0; pass < 32 / kDigitBits; ++pass) {
        const float *sk = pass & 1 ? k1 : k0;
        const int *si = pass & 1 ? i1 : i0;
        float *dk = pass & 1 ? k0 : k1;
        int *di = pass & 1 ? i0 : i1;
        reinterpret_cast<uint4 *>(hist)[tid] = make_uint4(0u, 0u, 0u, 0u);   // kHistBytes = 16 per thread
        __syncthreads();
        int rank[kSegRows], dig[kSegRows];
#pragma unroll
        for (int r = 0; r < kSegRows; ++r) {
            if (r >= rows)
                break;
            const int i = base + 32 * r;
            dig[r] = i < m ? (int)(((~__float_as_uint(sk[i])) >> (pass * kDigitBits)) & (kDigits - 1)) : kDigits;
            const unsigned int peers = __match_any_sync(0xffffffffu, dig[r]);
            const int below = __popc(peers & ((1u << lane) - 1u));
            unsigned short *slot = hist + dig[r] * kSampWarps + warp;
            int seen = 0;
            if (dig[r] < kDigits)
                seen = *slot;
            __syncwarp();
            if (dig[r] < kDigits && below == 0)
                *slot = (unsigned short)(seen + __popc(peers));
            __syncwarp();
            rank[r] = seen + below;
        }
        __syncthreads();
        // exclusive scan of the counts, digit-major: thread t owns counters 8 t .. 8 t + 7
        uint4 h = reinterpret_cast<uint4 *>(hist)[tid];
        unsigned int hw[4] = {h.x, h.y, h.z, h.w};
        int sum = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            sum += (int)(hw[q] & 0xffffu) + (int)(hw[q] >> 16);
        int total;
        int at = block_exclusive_scan(sum, warp_sums, total);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int lo = at, hi = at + (int)(hw[q] & 0xffffu);
            at = hi + (int)(hw[q] >> 16);
            hw[q] = (unsigned)lo | ((unsigned)hi << 16);
        }
        reinterpret_cast<uint4 *>(hist)[tid] = make_uint4(hw[0], hw[1], hw[2], hw[3]);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSegRows; ++r) {
            if (r >= rows)
                break;
            const int i = base + 32 * r;
            if (i < m) {
                const int to = (int)hist[dig[r] * kSampWarps + warp] + rank[r];
                dk[to] = sk[i];
                di[to] = si[i];
            }
        }
        __syncthreads();
    }
}

}  // namespace

__global__ void __cluster_dims__(kSampCtas, 1, 1) __launch_bounds__(kSampThreads, 1) sample_kernel(const __grid_constant__ SampleParams sp)
{
    extern __shared__ __align__(16) unsigned char ssm[];
    __shared__ int warp_sums[kSampWarps];
    __shared__ float s_red[kSampWarps];
    __shared__ float s_max[kSampCtas], s_sum, s_least;
    __shared__ int s_cnt[kSampCtas], s_pick;
    __shared__ ScanShared scan;

    cg::cluster_group cl = cg::this_cluster();
    const int me = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = sp.n;
    const int chunk = (n + kSampCtas - 1) / kSampCtas, chunk4 = (chunk + 3) & ~3;
    const int c0 = min(n, me * chunk), mine = min(n, c0 + chunk) - c0;      // this block's share of the vocabulary
    float *vals = reinterpret_cast<float *>(ssm);                            // block 0: n values; second buffer of the sort
    float *fk = vals + ((n + 3) & ~3);                                       // sorted candidates of this block
    int *fi = reinterpret_cast<int *>(fk + chunk4);
    unsigned short *hist = reinterpret_cast<unsigned short *>(fi + chunk4);
    float *vals0 = cl.map_shared_rank(vals, 0);

    // ---- logits / temperature, their maximum (Run.java:645-652, FindMax.call)
    float v[kSampRows];
    float mx = -FLT_MAX;
#pragma unroll
    for (int k = 0; k < kSampRows; ++k) {
        const int i = tid + k * kSampThreads;
        v[k] = 0.f;
        if (i < mine) {
            v[k] = __fdiv_rn(sp.logits[c0 + i], sp.temperature);
            mx = fmaxf(mx, v[k]);
        }
    }
    mx = warp_max(mx);
    if (lane == 0)
        s_red[warp] = mx;
    __syncthreads();
    mx = warp_max(s_red[lane]);
    cl.sync();                                   // every block of the cluster has started: its shared memory may be written
    if (tid < kSampCtas)
        cl.map_shared_rank(s_max, tid)[me] = mx;
    cl.sync();
    mx = s_max[0];
#pragma unroll
    for (int c = 1; c < kSampCtas; ++c)
        mx = fmaxf(mx, s_max[c]);
    // ---- exp in double, one sequential float sum, division (ExpSumNormalize.call, ExpSumNormalize.java:25-38)
#pragma unroll
    for (int k = 0; k < kSampRows; ++k) {
        const int i = tid + k * kSampThreads;
        if (i < mine) {
            v[k] = (float)exp((double)__fsub_rn(v[k], mx));
            vals0[c0 + i] = v[k];
        }
    }
    cl.sync();
    if (me == 0) {
        float sum = 0.0f;
        sequential_sum(vals, n, sum, INFINITY, false, scan);
        if (tid < kSampCtas)
            *cl.map_shared_rank(&s_sum, tid) = sum;
    }
    cl.sync();
    const float sum = s_sum;
#pragma unroll
    for (int k = 0; k < kSampRows; ++k) {
        const int i = tid + k * kSampThreads;
        if (i < mine) {
            if (sum != 0.0f)
                v[k] = __fdiv_rn(v[k], sum);
            sp.logits[c0 + i] = v[k];            // the reference turns the logits into probabilities in place
        }
    }

    unsigned long long rng = sp.st->rng;
    if ((double)sp.topp > 0.999) {   // Run.java:658 compares the float with the double literal
        // ---- Sampler.sample (Sampler.java:33-44)
#pragma unroll
        for (int k = 0; k < kSampRows; ++k) {
            const int i = tid + k * kSampThreads;
            if (i < mine)
                vals0[c0 + i] = v[k];
        }
        cl.sync();
        if (me == 0) {
            const float r = rng_next_float(rng);
            float cdf = 0.0f;
            const int hit = sequential_sum(vals, n, cdf, r, false, scan);
            if (tid == 0) {
                sp.st->rng = rng;
                sp.st->token = hit >= 0 ? hit : n - 1;
            }
        }
        return;
    }
    // ---- Sampler.sample_topp (Sampler.java:76-120): candidates in index order
    const int cur = sp.st->cur;
    const float *src_p = sp.prob[cur];
    const int *src_i = sp.index[cur];
    float *dst_p = sp.prob[cur ^ 1];
    int *dst_i = sp.index[cur ^ 1];
    const float cutoff = __fdiv_rn(__fsub_rn(1.0f, sp.topp), (float)(n - 1));
    int m = 0;
#pragma unroll
    for (int k = 0; k < kSampRows; ++k) {
        if (k * kSampThreads >= mine)
            break;
        const int i = tid + k * kSampThreads;
        const bool take = i < mine && v[k] >= cutoff;
        int total;
        const int at = m + block_exclusive_scan(take ? 1 : 0, warp_sums, total);
        if (take) {
            fk[at] = v[k];
            fi[at] = c0 + i;
        }
        m += total;
    }
    __syncthreads();
    sort_local(fk, fi, vals, reinterpret_cast<int *>(vals) + chunk, m, hist, warp_sums);
    if (tid < kSampCtas)
        cl.map_shared_rank(s_cnt, tid)[me] = m;
    cl.sync();
    // ---- places in the stable sort of the whole array: equal probabilities keep their order, which is the order of
    // the blocks' shares, then of the old tail
    int cnt[kSampCtas];
    int n0 = 0, longest = 0;
#pragma unroll
    for (int c = 0; c < kSampCtas; ++c) {
        cnt[c] = s_cnt[c];
        n0 += cnt[c];
        longest = max(longest, cnt[c]);
    }
    if (warp == 0) {
        float least = INFINITY;
        if (lane < kSampCtas && s_cnt[lane] > 0)
            least = cl.map_shared_rank(fk, lane)[s_cnt[lane] - 1];
        least = -warp_max(-least);
        if (lane == 0)
            s_least = least;
    }
    __syncthreads();
    const int search_steps = 32 - __clz(longest);
    for (int r = tid; r < m; r += kSampThreads) {
        const float pv = fk[r];
        int lo[kSampCtas], hi[kSampCtas];
#pragma unroll
        for (int c = 0; c < kSampCtas; ++c) {
            lo[c] = c == me ? r : 0;
            hi[c] = c == me ? r : cnt[c];
        }
        for (int s = 0; s < search_steps; ++s) {
#pragma unroll
            for (int c = 0; c < kSampCtas; ++c) {
                if (lo[c] < hi[c]) {
                    const int mid = (lo[c] + hi[c]) >> 1;
                    const float x = cl.map_shared_rank(fk, c)[mid];
                    if (x > pv || (c < me && x == pv))
                        lo[c] = mid + 1;
                    else
                        hi[c] = mid;
                }
            }
        }
        int to = 0;
#pragma unroll
        for (int c = 0; c < kSampCtas; ++c)
            to += lo[c];
        int tl = n0, th = n;                     // entries of the old tail in front of it: the larger ones
        if (tl < th && !(src_p[tl] > pv))
            th = tl;
        while (tl < th) {
            const int mid = (tl + th) >> 1;
            if (src_p[mid] > pv)
                tl = mid + 1;
            else
                th = mid;
        }
        to += tl - n0;
        dst_p[to] = pv;
        dst_i[to] = fi[r];
        if (to < n0)
            vals0[to] = pv;
    }
    const float least = s_least;
    for (int j = n0 + me * kSampThreads + tid; j < n; j += kSampCtas * kSampThreads) {
        const float pv = src_p[j];
        int to = j;                              // behind all candidates unless one is smaller
        if (pv > least) {
            to = j - n0;
            for (int c = 0; c < kSampCtas; ++c) {
                const float *list = cl.map_shared_rank(fk, c);
                int lo = 0, hi = cnt[c];
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (list[mid] >= pv)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                to += lo;
            }
        }
        dst_p[to] = pv;
        dst_i[to] = src_i[j];
        if (to < n0)
            vals0[to] = pv;
    }
    cl.sync();
    if (me != 0)
        return;
    // ---- the cumulative cut and the draw (Sampler.java:92-119)
    float cumulative = 0.0f;
    int last_idx = sequential_sum(vals, n0, cumulative, sp.topp, true, scan);
    if (last_idx < 0)
        last_idx = n0 - 1;
    const float r = __fmul_rn(rng_next_float(rng), cumulative);
    if (tid == 0)
        s_pick = n0 > 0 ? last_idx : -1;
    __syncthreads();
    // the running sums do not fall: the first that exceeds r is the one whose predecessor does not
    for (int i = tid; i <= last_idx; i += kSampThreads)
        if (r < vals[i] && (i == 0 || !(r < vals[i - 1])))
            s_pick = i;
    __syncthreads();
    if (tid == 0) {
        sp.st->rng = rng;
        sp.st->token = s_pick >= 0 ? dst_i[s_pick] : 0;
        sp.st->cur = cur ^ 1;
    }
}

// Values of the whole vocabulary (block 0; the sort's second buffer elsewhere), sorted candidates and their indices,
// digit counts of the local sort.
size_t sample_smem_bytes(int n)
{
    const int chunk = (n + kSampCtas - 1) / kSampCtas;
    return (size_t)((n + 3) & ~3) * 4 + (size_t)((chunk + 3) & ~3) * 8 + kHistBytes;
}

int sample_max_vocab(size_t smem_limit)
{
    int n = kSampMaxVocab;
    while (n > 0 && sample_smem_bytes(n) > smem_limit)
        n -= kSampCtas;
    return n;
}

// The limit belongs to the kernel on the device, whichever context asks for it: it is the same for all of them.
cudaError_t prepare_sampler()
{
    return cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sample_smem_bytes(kSampMaxVocab));
}

cudaError_t launch_sample(cudaStream_t stream, const SampleParams &sp)
{
    sample_kernel<<<kSampCtas, kSampThreads, sample_smem_bytes(sp.n), stream>>>(sp);
    return cudaGetLastError();
}

}  // namespace l2j
