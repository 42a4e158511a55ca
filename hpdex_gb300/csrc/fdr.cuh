// fdr.cuh -- the DE driver's post-processing on the device (sm_103a): Benjamini-Hochberg
// adjusted p-values over all (gene, target) tests, and fold changes from group means.
//
// BH follows scipy.stats.false_discovery_control(ps, method="bh"), which the reference DE
// driver calls (AI4Cell/hpdex src/hpdex/de.py:174-184): sort the p-values ascending, multiply
// the i-th (1-based) by m / i (one division, one multiplication, both rounded to nearest),
// replace each by the minimum of itself and everything after it, restore the input order,
// clip to [0, 1]. Equal p-values end with equal adjusted values whatever their order among
// themselves (the suffix minimum spans their whole run), so the sort need not match numpy's.
//
// The sort is a stable LSD radix sort of the p-values' bit patterns (non-negative doubles
// order like their bits) with 32-bit indices: 8 passes of 8-bit digits, each a count kernel
// (digit counts of every tile of entries), a scan kernel (one block per digit: prefix over
// the tiles) and a scatter kernel (per-warp stable ranks from warp match, the tile put in digit
// order in shared memory, then written as runs). At 4 million p-values everything stays in L2
// and a pass is bound by instruction issue. Per pass, before and after the tiles grew from 2,048
// entries written where they stood, and the scan from one block that read all counts with a
// stride: count 13 -> 12 us, scan 439 -> 6 us, scatter 69 -> 46 us; the whole call 4.69 -> 1.01 ms.
#pragma once
#include <cstdint>

#include "common.cuh"

namespace hpdex {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
// ITEMS entries per thread: tiles of 4,096 entries (16) for many p-values, of 1,024 (4) up to
// kSortSmall, where a pass is the time of one tile. A call with tiles of 1,024 / 2,048 / 4,096: 5,000
// p-values 163 / 183 / 224 us, 60,000 175 / 209 / 253, 500,000 262 / 274 / 294, 1,500,000 483 / 464 / 492, 4,000,000
// 1,023 / 977 / 970.
constexpr long long kSortSmall = 1ll << 19;

// -0.0 would sort after every positive value by its bits: it reads as +0.0 (they compare equal).
__device__ __forceinline__ unsigned long long sort_key(unsigned long long k) {
    return k == 0x8000000000000000ull ? 0ull : k;
}

// counts[d * ntiles + t]: entries of tile t with digit d.
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads) radix_count_kernel(const unsigned long long* keys,
                                                                   long long n, int shift,
                                                                   uint32_t* counts, int ntiles) {
    __shared__ uint32_t hist[256];
    hist[threadIdx.x] = 0u;
    __syncthreads();
    const long long t0 = (long long)blockIdx.x * (kSortThreads * ITEMS);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const long long i = t0 + (long long)k * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&hist[(uint32_t)(sort_key(keys[i]) >> shift) & 255u], 1u);
    }
    __syncthreads();
    counts[(size_t)threadIdx.x * ntiles + blockIdx.x] = hist[threadIdx.x];
}

// One block per digit: its row of counts becomes the exclusive prefix over the tiles, its sum
// goes to totals[digit].
__global__ void __launch_bounds__(kSortThreads) radix_scan_kernel(uint32_t* counts, int ntiles,
                                                                  uint32_t* totals) {
    __shared__ uint32_t ws[kSortWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* row = counts + (size_t)blockIdx.x * ntiles;
    uint32_t run = 0;
    for (int t = 0; t < ntiles; t += kSortThreads) {
        const int i = t + (int)threadIdx.x;
        const uint32_t v = i < ntiles ? row[i] : 0u;
        const uint32_t incl = warp_incl_scan(v);
        if (lane == 31) ws[warp] = incl;
        __syncthreads();
        uint32_t before = run, all = 0;
        for (int w = 0; w < kSortWarps; ++w) {
            if (w < warp) before += ws[w];
            all += ws[w];
        }
        if (i < ntiles) row[i] = before + incl - v;
        run += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = run;
}

// Stable scatter of one pass. vin == nullptr: the values are the input positions. Dynamic shared
// memory: kSortScatterSmem<ITEMS> bytes.
template <int ITEMS>
constexpr size_t kSortScatterSmem = (size_t)kSortThreads * ITEMS * 12 + kSortWarps * 256 * 4;
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(
    const unsigned long long* kin, const uint32_t* vin, unsigned long long* kout, uint32_t* vout,
    long long n, int shift, const uint32_t* offsets, const uint32_t* totals, int ntiles) {
    extern __shared__ __align__(16) unsigned char sort_smem[];
    unsigned long long* skey = reinterpret_cast<unsigned long long*>(sort_smem);
    uint32_t* sval = reinterpret_cast<uint32_t*>(skey + (kSortThreads * ITEMS));
    uint32_t(*whist)[256] = reinterpret_cast<uint32_t(*)[256]>(sval + (kSortThreads * ITEMS));
    __shared__ uint32_t gofs[256];  // where the tile's first entry of a digit goes, minus its place
                                    // in the tile's digit order
    __shared__ uint32_t ws[2][kSortWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int d = threadIdx.x; d < kSortWarps * 256; d += kSortThreads) (&whist[0][0])[d] = 0u;
    __syncthreads();
    // warp w takes the tile's w-th part of 32 * ITEMS entries, 32 consecutive ones per round
    const long long base = (long long)blockIdx.x * (kSortThreads * ITEMS) + (long long)warp * 32 * ITEMS;
    unsigned long long key[ITEMS];
    uint32_t place[ITEMS];  // digit << 16 | rank among the warp's entries of the digit
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const long long i = base + r * 32 + lane;
        key[r] = i < n ? sort_key(kin[i]) : 0ull;
    }
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const bool ok = base + r * 32 + lane < n;
        const uint32_t dig = ok ? ((uint32_t)(key[r] >> shift) & 255u) : 256u;
        const unsigned peers = __match_any_sync(0xffffffffu, dig);
        const uint32_t before = ok ? whist[warp][dig] : 0u;
        place[r] = (dig << 16) | (before + __popc(peers & lt));
        __syncwarp();
        if (ok && (peers & lt) == 0u) whist[warp][dig] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {   // thread d, digit d: the tile's count, where it starts in the tile and in the output
        const int d = threadIdx.x;
        uint32_t cnt = 0;
        for (int w = 0; w < kSortWarps; ++w) cnt += whist[w][d];
        const uint32_t tot = totals[d];
        const uint32_t ic = warp_incl_scan(cnt), it = warp_incl_scan(tot);
        if (lane == 31) { ws[0][warp] = ic; ws[1][warp] = it; }
        __syncthreads();
        uint32_t start = ic - cnt, out = it - tot;
        for (int w = 0; w < warp; ++w) { start += ws[0][w]; out += ws[1][w]; }
        gofs[d] = out + offsets[(size_t)d * ntiles + blockIdx.x] - start;
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = whist[w][d];
            whist[w][d] = start;
            start += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const long long i = base + r * 32 + lane;
        if (i < n) {
            const uint32_t pos = whist[warp][place[r] >> 16] + (place[r] & 0xffffu);
            skey[pos] = key[r];
            sval[pos] = vin ? vin[i] : (uint32_t)i;
        }
    }
    __syncthreads();
    const int cnt = (int)min((long long)(kSortThreads * ITEMS), n - (long long)blockIdx.x * (kSortThreads * ITEMS));
#pragma unroll 4
    for (int j = threadIdx.x; j < cnt; j += kSortThreads) {
        const unsigned long long k = skey[j];
        const uint32_t pos = gofs[(uint32_t)(k >> shift) & 255u] + (uint32_t)j;
        kout[pos] = k;
        vout[pos] = sval[j];
    }
}

// BH, step 1: per block of sorted p-values, the minimum of the adjusted values p_(i) * (m / i).
__device__ __forceinline__ double bh_adjusted(const unsigned long long* sk, long long i, long long m) {
    const double p = __longlong_as_double((long long)sk[i]);
    return __dmul_rn(p, __ddiv_rn((double)m, (double)(i + 1)));
}

// They are kept in adj (the division takes the narrow FP64 pipe: at 4 million values computing
// them in both this kernel and bh_apply_kernel took 107 + 119 us, once 81 + 52 us).
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads) bh_block_min_kernel(const unsigned long long* sk,
                                                                     long long m, double* adj,
                                                                     double* agg, uint32_t* bad) {
    __shared__ unsigned long long ws[kSortWarps];
    const long long t0 = (long long)blockIdx.x * (kSortThreads * ITEMS);
    unsigned long long v = 0x7ff0000000000000ull;  // +inf; non-negative doubles order like their bits
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const long long i = t0 + (long long)k * kSortThreads + threadIdx.x;
        if (i < m) {
            if (sk[i] > 0x3ff0000000000000ull) atomicOr(bad, 1u);  // NaN, negative or above 1
            const double x = bh_adjusted(sk, i, m);
            adj[i] = x;
            v = min(v, (unsigned long long)__double_as_longlong(x));
        }
    }
    v = warp_min(v);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long a = ws[0];
        for (int w = 1; w < kSortWarps; ++w) a = min(a, ws[w]);
        agg[blockIdx.x] = __longlong_as_double((long long)a);
    }
}

// BH, step 2 (one block): carry[b] = min(agg[b+1..]) (+inf for the last block).
__global__ void __launch_bounds__(1024) bh_carry_kernel(const double* agg, int nblocks, double* carry) {
    __shared__ double ws[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = (nblocks + 1023) / 1024;
    // thread t owns blocks [t*per, (t+1)*per), scanned from the end
    const int beg = min(nblocks, tid * per), end = min(nblocks, beg + per);
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    double s = inf;
    for (int b = beg; b < end; ++b) s = fmin(s, agg[b]);
    // suffix min over threads: thread t needs min over threads > t
    double incl = s;  // reverse inclusive scan within the warp
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_down_sync(0xffffffffu, incl, o);
        if (lane + o < 32) incl = fmin(incl, x);
    }
    if (lane == 0) ws[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        double v = ws[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const double x = __shfl_down_sync(0xffffffffu, v, o);
            if (lane + o < 32) v = fmin(v, x);
        }
        ws[lane] = v;  // min over warps >= lane
    }
    __syncthreads();
    // min over threads after t: later lanes of this warp, then later warps
    double after = __shfl_down_sync(0xffffffffu, incl, 1);
    if (lane == 31) after = inf;
    if (warp + 1 < 32) after = fmin(after, ws[warp + 1]);
    double run = after;
    for (int b = end - 1; b >= beg; --b) {
        carry[b] = run;
        run = fmin(run, agg[b]);
    }
}

// BH, step 3: suffix minimum inside each block plus its carry, clip, back to input order. The
// tile goes through shared memory, so that global accesses are by neighbouring threads while a
// thread scans ITEMS neighbouring values (one pad word after each keeps the banks apart); the values
// are compared as integers (non-negative doubles), which leaves the narrow FP64 pipe out.
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads) bh_apply_kernel(const double* adj,
                                                                 const uint32_t* sv, long long m,
                                                                 const double* carry, double* fdr) {
    using U = unsigned long long;
    __shared__ U tile[kSortThreads * (ITEMS + 1)];
    __shared__ U ws[kSortWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long t0 = (long long)blockIdx.x * (kSortThreads * ITEMS);
    const U inf = 0x7ff0000000000000ull;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int j = k * kSortThreads + (int)threadIdx.x;
        tile[j + j / ITEMS] = t0 + j < m ? (U)__double_as_longlong(adj[t0 + j]) : inf;
    }
    __syncthreads();
    U* mine = tile + (int)threadIdx.x * (ITEMS + 1);
    U tmin = inf;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) tmin = min(tmin, mine[k]);
    // min over the threads after this one (tile order = thread order)
    U incl = tmin;
    for (int o = 1; o < 32; o <<= 1) {
        const U x = __shfl_down_sync(0xffffffffu, incl, o);
        if (lane + o < 32) incl = min(incl, x);
    }
    if (lane == 0) ws[warp] = incl;
    __syncthreads();
    U after = __shfl_down_sync(0xffffffffu, incl, 1);
    if (lane == 31) after = inf;
    for (int w = warp + 1; w < kSortWarps; ++w) after = min(after, ws[w]);
    after = min(after, (U)__double_as_longlong(carry[blockIdx.x]));
#pragma unroll
    for (int k = ITEMS - 1; k >= 0; --k) {
        after = min(after, mine[k]);
        mine[k] = min(after, (U)0x3ff0000000000000ull);  // at most 1
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int j = k * kSortThreads + (int)threadIdx.x;
        if (t0 + j < m) fdr[sv[t0 + j]] = __longlong_as_double((long long)tile[j + j / ITEMS]);
    }
}

// Fold change and log2 fold change per (target, gene) from per-(gene, group) means
// (gene-major [gene * G + g], g = 0 the reference), as the reference DE driver computes them
// (de.py:138-142): fc = tar / ref; ref < 1e-10 -> clip; then tar < 1e-10 -> 1 / clip.
__global__ void fold_change_kernel(const double* means, long long n_genes, int G, double clip,
                                   double* fold, double* log2fold) {
    const long long n = (long long)(G - 1) * n_genes;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const long long t = i / n_genes, c = i - t * n_genes;
        const double ref = means[c * G], tar = means[c * G + t + 1];
        double f = __ddiv_rn(tar, ref);
        if (ref < 1e-10) f = clip;
        if (tar < 1e-10) f = __ddiv_rn(1.0, clip);
        fold[i] = f;
        log2fold[i] = log2(f);
    }
}

}  // namespace hpdex
