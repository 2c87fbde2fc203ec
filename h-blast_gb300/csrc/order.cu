// order.cu -- the ordering pass and the database/lookup-hit counters.
//
// The word finder appends HSPs in whatever order warps finish; H-BLAST fixes
// its order on the host (memory_defrag, h_blast.cu:1160-1208).  Here one
// cooperative kernel orders them by (query, subject, subject offset, query
// offset) -- per query and subject, the order in which NCBI's CPU word finder
// creates them (NF/blast_engine.c:553-576 feeds that list to BlastSaveInitHsp)
// -- writes the ordered records and the per-query ranges, and counts the lookup
// hits.  All sizes are read from device memory, so the pass needs no host round
// trip.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"

namespace hbg {

namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kOrderThreads = 1024;
constexpr int kWarps = kOrderThreads / 32;
// Up to kRankMax HSPs every one is ranked against all others; up to kRankAlone
// the same counts give the per-query ranges, and no CTA waits for another.
constexpr int kRankAlone = 1024;
constexpr int kRankMax = 16384;
constexpr int kItems = 8;                     // per thread and scatter round
constexpr int kRound = kOrderThreads * kItems;
constexpr int kPart = 1024;                   // fewest items worth a CTA of the radix sort (8192: 130 us for 16,000, 1024: 73)
constexpr int kSpinLimit = 1 << 22;           // polls of the grid barrier before it gives up

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned r;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(r));
    return r;
}

struct OrderSmem {
    uint32_t base[256];                       // next place of a digit's items of this CTA
    uint32_t scan[8];
    int ok, pad;
    union {
        uint64_t keys[kRankMax];
        struct {
            uint32_t cnt[kWarps][256];        // items of a digit in a warp, then before it in the round
            uint32_t before[4][256], total[4][256];
        } r;
    };
};
extern __shared__ __align__(16) unsigned char g_order_smem[];

__device__ __forceinline__ uint64_t key_of(const OrderArgs &a, const hbg_hsp &h) {
    uint64_t k = (uint64_t)(uint32_t)h.query;
    k = (k << a.bits_s) | (uint64_t)(uint32_t)h.subject;
    k = (k << a.bits_so) | (uint64_t)(uint32_t)h.s_off;
    return (k << a.bits_qo) | (uint64_t)(uint32_t)h.q_off;
}

// Every one of the first `grid` CTAs of the (cooperative) grid arrives before any leaves.  A wait that
// exceeds its limit reports through *error and the kernel ends.
__device__ bool grid_barrier(const OrderArgs &a, OrderSmem &sm, int grid, unsigned long long &target) {
    target += grid;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        sm.ok = 1;
        atomicAdd(a.barrier, 1ull);
        int polls = 0;
        unsigned long long seen;
        do {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(a.barrier) : "memory");
        } while (seen < target && ++polls < kSpinLimit);
        if (seen < target) {
            sm.ok = 0;
            atomicExch(a.error, 1ull);
        }
    }
    __syncthreads();
    __threadfence();
    return sm.ok != 0;
}

// An HSP's place among all n <= kRankAlone is the number of smaller keys; keys
// are distinct (a second hit starts one extension).  The same count for the
// bounds of its query and of its subject tells whether it is the first or last
// of them.
__device__ void rank_alone(const OrderArgs &a, OrderSmem &sm, int n) {
    const int lane = threadIdx.x & 31;
    if ((int)blockIdx.x * kWarps >= n)
        return;
    for (int i = threadIdx.x; i < n; i += kOrderThreads)
        sm.keys[i] = key_of(a, a.in[i]);
    __syncthreads();
    const int shift_s = a.bits_so + a.bits_qo, shift_q = shift_s + a.bits_s;
    for (int i = blockIdx.x * kWarps + (threadIdx.x >> 5); i < n; i += gridDim.x * kWarps) {
        const uint64_t key = sm.keys[i];
        // smallest and largest key of this query (one query: its key has no bits)
        const uint64_t q0 = a.bits_q ? (key >> shift_q) << shift_q : 0ull;
        const uint64_t q1 = a.bits_q ? q0 | ((1ull << shift_q) - 1ull) : ~0ull;
        const uint64_t s0 = (key >> shift_s) << shift_s;
        int below = 0, below_q = 0, upto_q = 0, below_s = 0;
        for (int j = lane; j < n; j += 32) {
            const uint64_t k = sm.keys[j];
            below += k < key;
            below_q += k < q0;
            upto_q += k <= q1;
            below_s += k < s0;
        }
        below = __reduce_add_sync(kAll, below);
        below_q = __reduce_add_sync(kAll, below_q);
        upto_q = __reduce_add_sync(kAll, upto_q);
        below_s = __reduce_add_sync(kAll, below_s);
        const int32_t *src = reinterpret_cast<const int32_t *>(a.in + i);
        int32_t *dst = reinterpret_cast<int32_t *>(a.out + below);
        if (lane < (int)(sizeof(hbg_hsp) / 4))
            dst[lane] = src[lane];
        if (a.q_first && lane == 0) {
            const int q = a.in[i].query;
            if (below == below_q)
                a.q_first[q] = (unsigned long long)below;
            if (below + 1 == upto_q)
                a.q_end[q] = (unsigned long long)upto_q;
            if (below == below_s)
                atomicAdd(a.q_passed + q, 1ull);
        }
    }
}

// The same for n <= kRankMax, two HSPs to a warp at a time; the ranges come from
// the ordered records, after a barrier.
__device__ void rank_all(const OrderArgs &a, OrderSmem &sm, int n) {
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < n; i += kOrderThreads)
        sm.keys[i] = key_of(a, a.in[i]);
    __syncthreads();
    const int step = gridDim.x * kWarps;
    for (int i = blockIdx.x * kWarps + (threadIdx.x >> 5); i < n; i += 2 * step) {
        const int i2 = i + step < n ? i + step : i;
        const uint64_t key = sm.keys[i], key2 = sm.keys[i2];
        int below = 0, below2 = 0;
#pragma unroll 4
        for (int j = lane; j < n; j += 32) {
            const uint64_t k = sm.keys[j];
            below += k < key;
            below2 += k < key2;
        }
        below = __reduce_add_sync(kAll, below);
        below2 = __reduce_add_sync(kAll, below2);
        if (lane < (int)(sizeof(hbg_hsp) / 4)) {
            reinterpret_cast<int32_t *>(a.out + below)[lane] = reinterpret_cast<const int32_t *>(a.in + i)[lane];
            reinterpret_cast<int32_t *>(a.out + below2)[lane] = reinterpret_cast<const int32_t *>(a.in + i2)[lane];
        }
    }
    if (!a.q_first)
        return;
    unsigned long long target = 0;
    if (!grid_barrier(a, sm, gridDim.x, target))
        return;
    for (int i0 = blockIdx.x * kOrderThreads; i0 < n; i0 += gridDim.x * kOrderThreads) {
        const int i = i0 + threadIdx.x;
        const bool on = i < n;
        int q = -1;
        bool fresh = false;
        if (on) {
            q = __ldcg(&a.out[i].query);
            const bool new_q = i == 0 || __ldcg(&a.out[i - 1].query) != q;
            if (new_q)
                a.q_first[q] = (unsigned long long)i;
            if (i == n - 1 || __ldcg(&a.out[i + 1].query) != q)
                a.q_end[q] = (unsigned long long)(i + 1);
            fresh = new_q || __ldcg(&a.out[i - 1].subject) != __ldcg(&a.out[i].subject);
        }
        const unsigned same = __match_any_sync(kAll, q);
        const unsigned cnt = __popc(__ballot_sync(kAll, fresh) & same);
        if (on && cnt && lane == __ffs(same) - 1)
            atomicAdd(a.q_passed + q, (unsigned long long)cnt);
    }
}

// Stable LSD radix sort, 8 bits a pass, over the key bits in use.  Each CTA
// owns a contiguous part of the items; a pass is a digit count per CTA, a grid
// barrier, the CTA's places from all counts, and the scatter.
__device__ void radix_all(const OrderArgs &a, OrderSmem &sm, int64_t n) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int grid = (int)min((int64_t)gridDim.x, (n + kPart - 1) / kPart);
    if ((int)blockIdx.x >= grid)
        return;
    const int64_t part = (n + grid - 1) / grid;
    const int64_t lo = min(n, part * (int64_t)blockIdx.x), hi = min(n, lo + part);
    const int bits = a.bits_q + a.bits_s + a.bits_so + a.bits_qo;
    unsigned long long target = 0;
    for (int64_t i = lo + t; i < hi; i += kOrderThreads) {
        a.keys[0][i] = key_of(a, a.in[i]);
        a.vals[0][i] = (uint32_t)i;
    }
    int src = 0;
    for (int shift = 0; shift < bits; shift += 8) {
        const uint64_t *kin = a.keys[src];
        const uint32_t *vin = a.vals[src];
        if (t < 256)
            sm.base[t] = 0;
        __syncthreads();               // (also: this CTA's first keys are written)
        for (int64_t i0 = lo; i0 < hi; i0 += kOrderThreads) {
            const int64_t i = i0 + t;
            const int dig = i < hi ? (int)((__ldcg(kin + i) >> shift) & 255u) : 256 + lane;
            const unsigned m = __match_any_sync(kAll, dig);
            if (dig < 256 && (m & lanemask_lt()) == 0)
                atomicAdd(&sm.base[dig], (uint32_t)__popc(m));
        }
        __syncthreads();
        if (t < 256)
            a.hist[blockIdx.x * 256 + t] = sm.base[t];
        if (!grid_barrier(a, sm, grid, target))
            return;
        {
            // places of this CTA's items of digit d: after all items of smaller
            // digits and after those of digit d in earlier CTAs
            const int d = t & 255, quarter = t >> 8;
            uint32_t before = 0, total = 0;
            for (int c = quarter; c < grid; c += 4) {
                const uint32_t x = __ldcg(a.hist + c * 256 + d);
                total += x;
                before += c < (int)blockIdx.x ? x : 0u;
            }
            sm.r.before[quarter][d] = before;
            sm.r.total[quarter][d] = total;
            __syncthreads();
            uint32_t tot = 0, bef = 0, incl = 0;
            if (t < 256) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    tot += sm.r.total[k][t];
                    bef += sm.r.before[k][t];
                }
                incl = tot;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t x = __shfl_up_sync(kAll, incl, o);
                    if (lane >= o)
                        incl += x;
                }
                if (lane == 31)
                    sm.scan[warp] = incl;
            }
            __syncthreads();
            if (t < 256) {
                uint32_t x = incl - tot + bef;
                for (int k = 0; k < warp; ++k)
                    x += sm.scan[k];
                sm.base[t] = x;
            }
        }
        uint64_t *kout = a.keys[src ^ 1];
        uint32_t *vout = a.vals[src ^ 1];
        for (int64_t r0 = lo; r0 < hi; r0 += kRound) {
            for (int i = t; i < kWarps * 256; i += kOrderThreads)
                (&sm.r.cnt[0][0])[i] = 0;
            __syncthreads();
            uint64_t key[kItems];
            uint32_t val[kItems], rank[kItems];
#pragma unroll
            for (int k = 0; k < kItems; ++k) {
                const int64_t i = r0 + (warp * kItems + k) * 32 + lane;
                const bool on = i < hi;
                key[k] = on ? __ldcg(kin + i) : 0;
                val[k] = on ? __ldcg(vin + i) : 0;
                const int dig = on ? (int)((key[k] >> shift) & 255u) : 256 + lane;
                const unsigned m = __match_any_sync(kAll, dig);
                const unsigned below = m & lanemask_lt();
                rank[k] = on ? sm.r.cnt[warp][dig] + (uint32_t)__popc(below) : 0xffffffffu;
                __syncwarp();
                if (on && below == 0)
                    sm.r.cnt[warp][dig] += (uint32_t)__popc(m);
                __syncwarp();
            }
            __syncthreads();
            if (t < 256) {
                uint32_t acc = sm.base[t];
#pragma unroll 4
                for (int w = 0; w < kWarps; ++w) {
                    const uint32_t x = sm.r.cnt[w][t];
                    sm.r.cnt[w][t] = acc;
                    acc += x;
                }
                sm.base[t] = acc;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < kItems; ++k)
                if (rank[k] != 0xffffffffu) {
                    const uint32_t pos = sm.r.cnt[warp][(key[k] >> shift) & 255u] + rank[k];
                    kout[pos] = key[k];
                    vout[pos] = val[k];
                }
            __syncthreads();
        }
        if (!grid_barrier(a, sm, grid, target))
            return;
        src ^= 1;
    }
    // the ordered records, and per query the range of its HSPs and the number
    // of subjects with at least one; whole warps step together, so that the
    // subject counts are summed per warp and query before the atomic
    const uint64_t *keys = a.keys[src];
    const uint32_t *vals = a.vals[src];
    const int shift_s = a.bits_so + a.bits_qo, shift_q = shift_s + a.bits_s;
    auto query_of = [&](uint64_t key) { return a.bits_q ? (int)(key >> shift_q) : 0; };
    for (int64_t i0 = lo; i0 < hi; i0 += kOrderThreads) {
        const int64_t i = i0 + t;
        const bool on = i < hi;
        int q = -1;
        bool fresh = false;
        if (on) {
            const uint64_t key = __ldcg(keys + i);
            const uint64_t prev = i > 0 ? __ldcg(keys + i - 1) : 0, next = i + 1 < n ? __ldcg(keys + i + 1) : 0;
            a.out[i] = a.in[__ldcg(vals + i)];
            q = query_of(key);
            const bool new_q = i == 0 || query_of(prev) != q;
            if (a.q_first) {
                if (new_q)
                    a.q_first[q] = (unsigned long long)i;
                if (i == n - 1 || query_of(next) != q)
                    a.q_end[q] = (unsigned long long)(i + 1);
            }
            fresh = new_q || (prev >> shift_s) != (key >> shift_s);
        }
        if (a.q_first) {
            const unsigned same = __match_any_sync(kAll, q);
            const unsigned cnt = __popc(__ballot_sync(kAll, fresh) & same);
            if (on && cnt && lane == __ffs(same) - 1)
                atomicAdd(a.q_passed + q, (unsigned long long)cnt);
        }
    }
}

// Lookup hits of a query: database count of each word times the entries the
// query has in its cell.
__device__ void count_hits(const OrderArgs &a, OrderSmem &sm) {
    for (int q = blockIdx.x; q < a.n_queries; q += gridDim.x) {
        const uint16_t *qc = a.query_cells + (size_t)q * HBG_NUM_CELLS;
        unsigned long long acc = 0;
        for (int w = threadIdx.x; w < HBG_NUM_CELLS; w += kOrderThreads) {
            const unsigned c = __ldg(qc + w);
            if (c)
                acc += __ldg(a.db_hist + w) * (unsigned long long)c;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            acc += __shfl_down_sync(kAll, acc, o);
        if ((threadIdx.x & 31) == 0)
            sm.keys[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < kWarps; ++k)
                acc += sm.keys[k];
            a.lookup_hits[q] = acc;
        }
        __syncthreads();
    }
}

// The ordering pass in one launch.  A dozen HSPs 9 us, 570 10 us, 9155 27 us
// (sorted: 72), 16,000 64 us, 50,000 115 us, 1.4 M 397 us; as 25 launches of
// separate passes 107, 130, 214, -, 237 and 893 us.  The sort is bound by its
// grid barriers and block-wide steps (ten us per 8 bits of the key) until the
// items are many.
__global__ void __launch_bounds__(kOrderThreads, 1) order_kernel(OrderArgs a) {
    OrderSmem &sm = *reinterpret_cast<OrderSmem *>(g_order_smem);
    count_hits(a, sm);
    const unsigned long long c = *a.count;
    const int64_t n = (int64_t)(c < (unsigned long long)a.cap ? c : (unsigned long long)a.cap);
    if (n <= kRankAlone)
        rank_alone(a, sm, (int)n);
    else if (n <= kRankMax)
        rank_all(a, sm, (int)n);
    else
        radix_all(a, sm, n);
}

// A warp spreads 1024 consecutive letters, a lane every 32nd: the subject of
// the first by bisection, the others from there.  Bound by the copy to the
// device: 18 M letters in 50,000 subjects open in 0.56 ms, 359 M in 1 M subjects
// in 10.3 ms; 13.2 and 288 ms with the checks and the staging on the host.
constexpr int kSpread = 1024;
__global__ void __launch_bounds__(256)
spread_letters(const uint8_t *raw, int64_t from, int64_t count, const int64_t *first, int32_t n, uint8_t *out,
               int32_t *bad) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
    for (int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 32; c * kSpread < count; c += warps) {
        const int64_t begin = from + c * kSpread, end = min(from + count, begin + kSpread);
        // the last subject that starts at or before `begin`
        int32_t lo = 0, hi = n;
        while (hi - lo > 1) {
            const int32_t mid = lo + (hi - lo) / 2;
            if (first[mid] <= begin)
                lo = mid;
            else
                hi = mid;
        }
        int32_t i = lo;
        int64_t next = first[i + 1];
        const int64_t shift = 1 - first[0];
        for (int64_t p = begin + lane; p < end; p += 32) {
            while (p >= next)
                next = first[++i + 1];
            const uint8_t a = raw[p - from];
            out[p + shift + i] = a;
            if (a == 0 || a >= HBG_ALPHABET)
                atomicMin(bad, i);
        }
    }
}

__global__ void __launch_bounds__(256)
db_histogram(const uint8_t *db, int64_t n, unsigned long long *hist) {
    extern __shared__ unsigned int hsm[];
    for (int i = threadIdx.x; i < HBG_NUM_CELLS; i += blockDim.x)
        hsm[i] = 0;
    __syncthreads();
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p + 2 < n;
         p += (int64_t)gridDim.x * blockDim.x) {
        const unsigned a = db[p], b = db[p + 1], c = db[p + 2];
        if (a && b && c)
            atomicAdd(&hsm[(a << 10) | (b << 5) | c], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < HBG_NUM_CELLS; i += blockDim.x)
        if (hsm[i])
            atomicAdd(hist + i, (unsigned long long)hsm[i]);
}

}  // namespace

int order_grid(int device) {
    int sms = 1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return std::min(sms, kOrderMaxGrid);
}

cudaError_t launch_order(const OrderArgs &a, int grid, cudaStream_t stream) {
    OrderArgs args = a;
    void *params[] = {&args};
    cudaError_t e = cudaFuncSetAttribute(order_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(OrderSmem));
    if (e != cudaSuccess)
        return e;
    return cudaLaunchCooperativeKernel((const void *)order_kernel, dim3((unsigned)grid), dim3(kOrderThreads), params,
                                       sizeof(OrderSmem), stream);
}

cudaError_t launch_spread_letters(const uint8_t *raw, int64_t from, int64_t count, const int64_t *first, int32_t n,
                                  uint8_t *out, int32_t *bad, cudaStream_t stream) {
    const int64_t ctas = (count + 8 * kSpread - 1) / (8 * kSpread);
    spread_letters<<<(unsigned)std::min<int64_t>(ctas, 65535), 256, 0, stream>>>(raw, from, count, first, n, out, bad);
    return cudaGetLastError();
}

cudaError_t launch_db_histogram(const uint8_t *db, int64_t n, unsigned long long *hist,
                                cudaStream_t stream) {
    const size_t smem = HBG_NUM_CELLS * sizeof(unsigned int);
    cudaError_t e = cudaFuncSetAttribute(db_histogram, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess)
        return e;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    db_histogram<<<sms > 0 ? sms : 1, 256, smem, stream>>>(db, n, hist);
    return cudaGetLastError();
}

}  // namespace hbg
