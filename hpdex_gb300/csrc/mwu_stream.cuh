// mwu_stream.cuh -- per-gene rank sums by streaming the targets past the sorted reference (sm_103a).
//
// Computes the same integers as mwu_rank_kernel (mwu_rank.cuh: doubled U2, tie sums, zero blocks,
// fused p-values) for float genes, without putting a gene's target elements in order. Only the
// reference elements, usually the smallest part of a gene, are sorted; a target element then
// needs no neighbour to know its place:
//   - A[g] += 2 * #ref{< x} + #ref{== x}, looked up in the sorted reference (a bucket table and
//     a short walk over the bucket's distinct values);
//   - with c0 = #ref{== x} and s elements of group g equal to x, the pair (x, g) adds
//     (c0+s)^3 - (c0+s) - (c0^3 - c0) to B[g]. Every element adds the share it would have alone
//     (s = 1), 3 c0^2 + 3 c0; pairs with s > 1 add the rest, 3 c0 (s^2 - s) + s^3 - s, once. They
//     are found by hashing: a bitmap marks the cells that (x, g) hits and a second one those hit
//     more than once; a second pass over the targets collects the elements of such cells (repeats,
//     and the few pairs that share a cell) and counts them in a table, in as many hash partitions
//     as it needs.
// The work per entry is the same for 37 groups of 400 elements and 1,500 of 20, and none of it
// depends on a slab of the gene fitting in shared memory, which holds the sorted reference, the
// accumulators and the table. A gene whose reference does not fit, whose reference values
// crowd a bucket or one of whose pairs occurs more than 65,535 times is listed for mwu_rank_kernel,
// launched behind this one.
//
// It gains where values seldom repeat: there mwu_rank_kernel resolves every bucket of several
// values pairwise (continuous data at 60,000 entries a gene: 5 times the time), while here only
// the first pass over a gene is bound by memory and the rest by instruction issue. Where a few
// values hold most elements its second pass costs more than the one-value buckets of
// mwu_rank_kernel (1,000 genes of 10,000 entries and 20 groups, 100 steps of a normal: 0.31 against
// 0.21 ms). column_ties_kernel's sample and the plan's grouping (StreamRule) divide the genes.
#pragma once
#include "mwu_rank.cuh"

namespace hpdex {

struct StreamArgs {
    const RankTask* tasks;
    const int32_t* order;        // genes in processing order [n_order]
    const uint16_t* order_task;  // task of each entry of `order` (null: all task 0)
    int32_t n_order;
    int32_t* queue;              // work counter
    int32_t G;                   // layout G: the largest task G of the launch
    int32_t nb_max_log2;         // bucket table capacity: 8 entries per thread
    int32_t region;              // bytes for the reference and the table, a multiple of 16
    // per CTA a slice for the decoded targets of its gene: keys and groups (as in RankArgs)
    void* dk_global;
    void* dg_global;
    long long slice;
    const double* erfc_table;    // non-null: p-values too, as in RankArgs
    int32_t* left;               // genes (and tasks) left to mwu_rank_kernel, and how many
    uint16_t* left_task;
    int32_t* n_left;
};

constexpr int kStreamMaxBucket = 512;    // reference elements of a bucket of several values
constexpr uint32_t kStreamMinTable = 16u << 10;  // (a region is at least four of these)

// Reference elements that a region holds: their keys twice (as read, as scattered) and the ends of
// their runs, two paddings of 16 bytes. The bitmaps and the table come where the scattered keys
// were: at least 2/5 of a region of 4 * kStreamMinTable bytes, the smallest a launch has.
__host__ __device__ inline uint32_t stream_ref_cap(size_t region, size_t key_bytes) {
    return (uint32_t)((region - 64) / (2 * key_bytes + 2));
}

// Shared memory: accumulators (28 bytes per group: A and B as in mwu_rank_kernel, the stored and
// negative counts, and the targets' own shares of B in one word), bucket table, then the region.
__host__ __device__ inline size_t stream_acc_bytes(int G) { return RankSmem::align16((size_t)G * 28); }
__host__ __device__ inline size_t stream_bucket_bytes(int nb_log2) { return (((size_t)1 << nb_log2) + 8) * 4; }

// Exclusive prefix sum of x[0..L) in place, x[L] = total, *xmax = max x[i] (zeroed before);
// L <= 8 * NT, x 16-byte aligned.
template <int NT>
__device__ void block_scan_max(uint32_t* x, int L, uint32_t* ws, uint32_t* xmax) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int beg = min(L, tid * 8), cnt = min(L, beg + 8) - beg;
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = i < cnt ? x[beg + i] : 0u;
    uint32_t sum = 0, mx = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) { sum += v[i]; mx = max(mx, v[i]); }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0 && mx) atomicMax(xmax, mx);
    const uint32_t inc = warp_incl_scan(sum);
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    const uint32_t u = lane < NT / 32 ? ws[lane] : 0u;
    const uint32_t pu = warp_incl_scan(u);
    uint32_t o = __shfl_sync(0xffffffffu, pu - u, warp) + inc - sum;
    if (warp == 0 && lane == 31) x[L] = pu;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (i < cnt) x[beg + i] = o;
        o += v[i];
    }
    __syncthreads();
}

// Brings the whole 16-byte words of [b, e) to L2 (one thread; nothing is waited for).
__device__ __forceinline__ void l2_prefetch(const void* b, const void* e) {
    unsigned long long p = ((unsigned long long)b + 15ull) & ~15ull;
    const unsigned long long q = (unsigned long long)e & ~15ull;
    while (p < q) {
        const uint32_t n = (uint32_t)min(q - p, 1ull << 20);
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(n) : "memory");
        p += n;
    }
}

// Shared memory by 32-bit addresses (smem_addr): the passes over the elements keep one base
// address per array, where pointers would be converted at every access.
__device__ __forceinline__ uint32_t lds(uint32_t p) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(p));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t p) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(p));
    return v;
}
template <class K>
__device__ __forceinline__ K lds_key(uint32_t p) {
    if constexpr (sizeof(K) == 4) {
        return lds(p);
    } else {
        unsigned long long v;
        asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(p));
        return v;
    }
}
__device__ __forceinline__ void reds(uint32_t p, uint32_t v) {
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ors(uint32_t p, uint32_t v) {
    uint32_t old;
    asm volatile("atom.shared.or.b32 %0, [%1], %2;" : "=r"(old) : "r"(p), "r"(v) : "memory");
    return old;
}

// Hash of a (key, group) pair: the high bits choose the cell or slot, the low ones the partition.
// (Multipliers of MurmurHash3's finaliser and of xxHash.)
__device__ __forceinline__ uint32_t pair_hash(uint32_t key, uint32_t g) {
    uint32_t h = key * 0x85ebca6bu + g * 0x9e3779b1u;
    h ^= h >> 15;
    return h * 0xc2b2ae35u;
}
__device__ __forceinline__ uint32_t pair_hash(unsigned long long key, uint32_t g) {
    return pair_hash((uint32_t)key * 0x27d4eb2fu ^ (uint32_t)(key >> 32), g);
}

// A table of (key, group) pairs and their counts. Slot: high word the key (32-bit keys) or the
// element's place in the decoded copy (64-bit keys, read back there), low word group << 16 |
// count; groups of pairs are targets (> 0), so an empty slot is 0.
struct PairTable {
    unsigned long long* slot;
    uint32_t n;
};
template <class K>
__device__ __forceinline__ K slot_key(unsigned long long s, const K* dk) {
    if constexpr (sizeof(K) == 4) return (uint32_t)(s >> 32);
    else return dk[(uint32_t)(s >> 32)];
}
// Counts one element; false when the table has no room within the probe limit, or (`wide`: more elements
// are counted than a slot can hold) the pair's count leaves its 16 bits. (That count may have carried into the
// group; every other lookup still ends, and the caller drops the table.)
template <class K>
__device__ __forceinline__ bool pair_count(const PairTable& t, K key, uint32_t g, uint32_t entry,
                                           uint32_t h, const K* dk, bool wide) {
    const uint32_t id = sizeof(key) == 4 ? (uint32_t)key : entry;
    const unsigned long long mine = ((unsigned long long)id << 32) | (g << 16) | 1u;
    uint32_t p = __umulhi(h, t.n);
    for (int probe = 0; probe < 128; ++probe) {
        unsigned long long cur = *(volatile unsigned long long*)(t.slot + p);
        if (cur == 0ull) {
            cur = atomicCAS(t.slot + p, 0ull, mine);
            if (cur == 0ull) return true;
        }
        bool same;
        if constexpr (sizeof(key) == 4) same = (cur >> 16) == (mine >> 16);
        else same = (((uint32_t)cur >> 16) == g) && slot_key(cur, dk) == key;
        if (same) {
            uint32_t* count = reinterpret_cast<uint32_t*>(t.slot + p);
            if (wide) return (atomicAdd(count, 1u) & 0xffffu) != 0xffffu;
            red_add<true>(count, 1u);
            return true;
        }
        p = p + 1u == t.n ? 0u : p + 1u;
    }
    return false;
}

// How a column's values repeat, from kTieSample entries evenly spaced over it: `equal` of them equal an
// earlier one, and `repeat` is the share of their pairs that are equal (an estimate of the sum of
// squared frequencies of the column's values). Both 0 for columns of fewer than 2 * kTieSample entries; one
// block a column. The plan decides by both (StreamRule).
struct ColumnTies {
    float repeat;
    uint32_t equal;
};
constexpr int kTieSample = 512;
template <class V>
__global__ void __launch_bounds__(128) column_ties_kernel(const V* data, const int64_t* indptr, ColumnTies* ties) {
    using K = typename Val<V>::Key;
    __shared__ unsigned long long slot[2 * kTieSample];  // key + 1 (0: empty)
    __shared__ uint32_t more[2 * kTieSample];            // elements of the slot's value after its first
    __shared__ uint32_t equal, pairs, used;
    const long long b = indptr[blockIdx.x], n = indptr[blockIdx.x + 1] - b;
    if (n < 2 * kTieSample) {
        if (threadIdx.x == 0) ties[blockIdx.x] = ColumnTies{0.0f, 0u};
        return;
    }
    for (int i = threadIdx.x; i < 2 * kTieSample; i += 128) { slot[i] = 0ull; more[i] = 0u; }
    if (threadIdx.x == 0) { equal = 0u; pairs = 0u; used = 0u; }
    __syncthreads();
    for (int i = threadIdx.x; i < kTieSample; i += 128) {
        const V v = data[b + (long long)i * n / kTieSample];
        if (!Val<V>::finite(v) || Val<V>::zero(v)) continue;
        atomicAdd(&used, 1u);
        const unsigned long long k = (unsigned long long)Val<V>::key(v) + 1ull;
        uint32_t p = pair_hash((unsigned long long)k, 0u) >> 22;  // 1,024 slots, at most half taken
        for (;; p = (p + 1u) & (2u * kTieSample - 1u)) {
            const unsigned long long old = atomicCAS(&slot[p], 0ull, k);
            if (old == 0ull) break;
            if (old == k) {
                atomicAdd(&equal, 1u);
                atomicAdd(&pairs, atomicAdd(&more[p], 1u) + 1u);
                break;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0)
        ties[blockIdx.x] = ColumnTies{used > 1u ? 2.0f * (float)pairs / ((float)used * (float)(used - 1u)) : 0.0f, equal};
}

// One 1,024-thread CTA per SM takes genes from the work queue. Per gene:
//   entries    once from HBM (the next gene's are asked into L2 meanwhile): reference keys to shared
//              memory, the stored targets' keys and groups to the CTA's slice (6 or 10 bytes each,
//              L2), so that the passes below need no group gather and no test
//   reference  counted into buckets, scattered, ordered inside each bucket; equal values form runs
//   targets    four per thread and step: two reads of the bucket table, one of the bucket's first
//              value and run, adds to the group's sums, one bit of the bitmap
//   repeats    only if some cell was hit twice: the elements of such cells are first moved together,
//              then counted with whole warps (counted where they stood, a few lanes at a time, a
//              screen on this kernel took 3.50 ms, now 2.90, exact mode's data 2.10, now 2.01)
//   finalize   as in mwu_rank_kernel; p-values during the next gene's target pass
// Bound by instruction issue (2.4 of 4 a cycle) with the shared-memory atomics next: 512 or 768
// threads, or two CTAs' worth of registers, lose more to latency than they gain. Rank sums
// without the p-values of exact mode 4.94 -> 2.10 ms (60,000 x 4,000 dense, 1,500 groups of 3-40:
// 9% -> 14% of the copy bandwidth), dense doubles (20,011 x 1,501, 37 groups) 2.07 -> 0.68 ms; with
// the repeats moved together 2.01 and 0.62, with more buckets 1.78 (17% of the copy bandwidth) and 0.62.
template <class V, int NT>
__global__ void __launch_bounds__(NT, 1) mwu_stream_kernel(const StreamArgs a) {
    using K = typename Val<V>::Key;
    using GT = uint16_t;
    constexpr uint32_t kNoGroup = 0xffffu;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned long long s_tref;
    __shared__ uint32_t s_nref, s_ntar, s_neg, s_maxb, s_maxrun, s_bad, s_hits, s_cells;
    __shared__ int s_pv_gene, s_pv_task;  // gene whose p-values are pending (-1: none)
    __shared__ uint32_t s_pvq;            // its p-value tiles taken so far
    __shared__ int s_next_gene, s_next_task;
    __shared__ long long s_next_p0, s_next_p1;
    __shared__ unsigned long long s_next_kmin, s_next_kmax;
    __shared__ uint32_t s_next_hz;
    __shared__ uint32_t s_ws[32];
    __shared__ uint32_t s_mixed[8 * NT / 32];  // buckets of more than 32 reference elements that
                                               // hold several values

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int GL = a.G;
    unsigned long long* A = reinterpret_cast<unsigned long long*>(smem);
    unsigned long long* B = A + GL;
    uint32_t* nz = reinterpret_cast<uint32_t*>(B + GL);
    uint32_t* ng = nz + GL;
    uint32_t* b32s = ng + GL;
    // Sums that cannot leave 32 bits are kept as words, side by side: neighbouring groups then lie
    // in neighbouring banks, and no carry is looked at. (The target pass is bound by its shared-
    // memory atomics.)
    uint32_t* a32s = reinterpret_cast<uint32_t*>(A);
    // bucket table; the word before it stays 0, the start of the first bucket after the scatter
    uint32_t* bs = reinterpret_cast<uint32_t*>(smem + stream_acc_bytes(GL)) + 4;
    unsigned char* region = smem + stream_acc_bytes(GL) + stream_bucket_bytes(a.nb_max_log2);

    K* dk = reinterpret_cast<K*>(a.dk_global) + (size_t)blockIdx.x * a.slice;
    GT* dg = reinterpret_cast<GT*>(a.dg_global) + (size_t)blockIdx.x * a.slice;

    // Thread NT - 1 fetches the next gene in three steps, one per phase of the current gene (so that
    // it waits for none of the loads), and asks for its row ids and values to be brought to L2.
    int next_i = 0, next_c = -1, next_t = 0;
    auto fetch_index = [&]() { next_i = atomicAdd(a.queue, 1); };
    auto fetch_gene = [&]() {
        next_c = next_i < a.n_order ? a.order[next_i] : -1;
        next_t = next_i < a.n_order && a.order_task ? (int)a.order_task[next_i] : 0;
    };
    auto fetch_column = [&]() {
        s_next_gene = next_c;
        s_next_task = next_t;
        if (next_c < 0) return;
        const RankTask* t = a.tasks + next_t;
        const long long b = t->indptr[next_c], e = t->indptr[next_c + 1];
        l2_prefetch(t->rows + b, t->rows + e);
        l2_prefetch(reinterpret_cast<const V*>(t->data) + b, reinterpret_cast<const V*>(t->data) + e);
        s_next_p0 = b;
        s_next_p1 = e;
        s_next_kmin = t->col_kmin[next_c];
        s_next_kmax = t->col_kmax[next_c];
        s_next_hz = t->col_has_zero[next_c];
    };
    if (tid == NT - 1) { fetch_index(); fetch_gene(); fetch_column(); }
    if (tid == 0) { s_pv_gene = -1; s_pv_task = 0; s_pvq = 0u; bs[-1] = 0u; }
    __syncthreads();

    for (;;) {
        const int c = s_next_gene, ti = s_next_task;
        const int pv_c = s_pv_gene;
        const RankTask* pv_tk = (a.erfc_table && pv_c >= 0) ? a.tasks + s_pv_task : nullptr;
        if (c < 0) {
            if (pv_tk) pvalue_tiles(pv_tk, pv_c, &s_pvq, a.erfc_table);
            break;
        }
        const RankTask* tk = a.tasks + ti;
        const int G = tk->G, zh = tk->zero_handling;
        const GT* gidp = reinterpret_cast<const GT*>(tk->group_of_row);
        const uint32_t nrows = (uint32_t)tk->n_rows;
        const long long p0 = s_next_p0;
        const uint32_t nraw = (uint32_t)(s_next_p1 - p0);
        const int32_t* rows = tk->rows + p0;
        const V* data = reinterpret_cast<const V*>(tk->data) + p0;
        K kmin = (K)s_next_kmin, kmax = (K)s_next_kmax;
        if (zh == ZH_NONE && (s_next_hz & 1u)) {
            const K kz = Val<V>::key(V(0));
            kmin = kz < kmin ? kz : kmin;
            kmax = kz > kmax ? kz : kmax;
        }
        // four buckets per expected reference element, at least 2,048 (two to a thread): values crowd, so
        // that with two, and 64 at least, a target walked past the values before its own (exact
        // mode, 40 reference cells: 2.01 ms, now 1.78; 8,192 for every gene 1.81 and the screen 1%
        // slower for the longer clear and scan)
        const float expect = 4.0f * (float)nraw * (float)tk->group_rows[0] / (float)max(1u, nrows);
        int nbl = 11;
        while (nbl < a.nb_max_log2 && (float)(1u << nbl) < expect) ++nbl;
        const int NB = 1 << nbl;
        for (int g = tid; g < GL; g += NT) { A[g] = 0ull; B[g] = 0ull; nz[g] = 0u; ng[g] = 0u; b32s[g] = 0u; }
        for (int b = tid; b <= NB; b += NT) bs[b] = 0u;
        if (tid == 0) {
            s_tref = 0ull;
            s_nref = 0u; s_ntar = 0u; s_neg = 0u; s_maxb = 0u; s_maxrun = 0u; s_bad = 0u; s_hits = 0u; s_cells = 0u;
        }
        __syncthreads();
        if (tid == NT - 1) fetch_index();

        unsigned long long tref = 0ull;
        bool words_a = true;  // A is in a32s
        auto gene = [&](auto vm_tag) {
            constexpr bool VM = decltype(vm_tag)::value;
            BucketMap<V> bmap;
            bmap.setup(kmin, kmax, nbl);
            auto stored = [&](V v) { return Val<V>::finite(v) && (zh == ZH_NONE || !Val<V>::zero(v)); };
            auto bucket_start = [&](uint32_t b) { return bs[(int)b - 1]; };  // (after the scatter)

            // ---- the entries once: reference keys to the start of the region, the stored
            // targets' (key, group) to the CTA's slice ----
            K* stage = reinterpret_cast<K*>(region);
            const uint32_t cap = stream_ref_cap((size_t)a.region, sizeof(K));
            {
                // a warp's tile of 128: 4 entries per lane, neighbouring lanes on neighbouring
                // entries (a whole tile: no bounds to test)
                auto tile = [&](uint32_t t, auto whole_tag) {
                    constexpr bool WHOLE = decltype(whole_tag)::value;
                    const int32_t* rp = rows + t + lane;
                    const V* vp = data + t + lane;
                    int32_t r[4];
                    V v[4];
                    uint32_t g[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const bool in = WHOLE || t + 32u * k + lane < nraw;
                        r[k] = in ? __ldcs(rp + 32 * k) : -1;
                        v[k] = in ? ld_stream(vp + 32 * k) : V(0);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        g[k] = (uint32_t)r[k] < nrows ? (uint32_t)__ldg(gidp + r[k]) : kNoGroup;
                    unsigned m[4], q[4];
                    uint32_t nm = 0, nq = 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const bool st = g[k] != kNoGroup && stored(v[k]);
                        m[k] = __ballot_sync(0xffffffffu, st && g[k] == 0u);
                        q[k] = __ballot_sync(0xffffffffu, st && g[k] != 0u);
                        nm += __popc(m[k]);
                        nq += __popc(q[k]);
                    }
                    uint32_t pm = 0, pq = 0;
                    if (lane == 0) {
                        if (nm) pm = atomicAdd(&s_nref, nm);
                        pq = atomicAdd(&s_ntar, nq);
                    }
                    pm = __shfl_sync(0xffffffffu, pm, 0);
                    pq = __shfl_sync(0xffffffffu, pq, 0);
                    const unsigned below = (1u << lane) - 1u;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const K key = Val<V>::key(v[k]);
                        if ((q[k] >> lane) & 1u) {
                            const uint32_t o = pq + __popc(q[k] & below);
                            dk[o] = key;
                            dg[o] = (GT)g[k];
                        }
                        pq += __popc(q[k]);
                        if (m[k]) {
                            if ((m[k] >> lane) & 1u) {
                                const uint32_t o = pm + __popc(m[k] & below);
                                if (o < cap) stage[o] = key;
                                else s_bad = 1u;
                            }
                            pm += __popc(m[k]);
                        }
                    }
                };
                for (uint32_t t = 128u * (uint32_t)warp; t < nraw; t += 4u * NT) {
                    if (t + 128u <= nraw) tile(t, std::true_type{});
                    else tile(t, std::false_type{});
                }
            }
            __syncthreads();
            if (s_bad) return;
            const uint32_t nref = s_nref;
            const K k0 = Val<V>::key(V(0));
            {
                uint32_t neg = 0;
                for (uint32_t i = tid; i < nref; i += NT) {
                    const K key = stage[i];
                    red_add<true>(&bs[bmap.template at<VM>(key)], 1u);
                    neg += key < k0;
                }
                neg = __reduce_add_sync(0xffffffffu, neg);
                if (lane == 0 && neg) atomicAdd(&s_neg, neg);
            }
            __syncthreads();

            // ---- sorted: by bucket, then inside each bucket ----
            block_scan_max<NT>(bs, NB, s_ws, &s_maxb);
            K* mid = reinterpret_cast<K*>(region + RankSmem::align16(sizeof(K) * nref));
            uint16_t* run_end = reinterpret_cast<uint16_t*>(region + a.region - RankSmem::align16(2 * (size_t)nref + 2));
            for (uint32_t i = tid; i < nref; i += NT) {
                const K key = stage[i];
                mid[atom_add<true>(&bs[bmap.template at<VM>(key)], 1u)] = key;
            }
            const bool big = s_maxb > 32u;
            if (big)
                for (int i = tid; i < (NB + 31) / 32; i += NT) s_mixed[i] = 0u;
            __syncthreads();
            // (bs[b] has counted up to the end of bucket b)
            if (big) {
                for (uint32_t p = tid; p < nref; p += NT) {
                    const K key = mid[p];
                    const uint32_t b = bmap.template at<VM>(key);
                    if (mid[bucket_start(b)] != key) atomicOr(&s_mixed[b >> 5], 1u << (b & 31u));
                }
                __syncthreads();
            }
            // skey[j]: the reference in ascending order; run_end[j]: where the run of skey[j] ends,
            // so j is also the number of reference elements below skey[j]'s run when it starts there
            K* skey = stage;
            uint32_t longest = 0;
            for (uint32_t p = tid; p < nref; p += NT) {
                const K key = mid[p];
                const uint32_t b = bmap.template at<VM>(key);
                const uint32_t s = bucket_start(b), e = bs[b], m = e - s;
                if (m > 32u && !((s_mixed[b >> 5] >> (b & 31u)) & 1u)) {  // one value
                    skey[p] = key;
                    run_end[p] = (uint16_t)e;
                    if (p == s) tref += (unsigned long long)m * m * m - m;
                    longest = max(longest, m);
                    continue;
                }
                if (m > (uint32_t)kStreamMaxBucket) { s_bad = 1u; continue; }
                uint32_t lt = 0, eq = 0, before = 0;
                for (uint32_t j = s; j < e; ++j) {
                    const K kj = mid[j];
                    lt += kj < key;
                    eq += kj == key;
                    before += kj == key && j < p;
                }
                skey[s + lt + before] = key;
                run_end[s + lt + before] = (uint16_t)(s + lt + eq);
                if (before == 0u) tref += (unsigned long long)eq * eq * eq - eq;
                longest = max(longest, eq);
            }
            longest = __reduce_max_sync(0xffffffffu, longest);
            if (lane == 0) atomicMax(&s_maxrun, longest);
            __syncthreads();
            if (s_bad) return;
            // the place of a key in its bucket's reference [j, e): the elements before j are below it
            const uint32_t bs_at = smem_addr(bs), key_at = smem_addr(skey), end_at = smem_addr(run_end);
            auto ref_key = [&](uint32_t j) { return lds_key<K>(key_at + (uint32_t)sizeof(K) * j); };
            auto walk = [&](K key, uint32_t& j, uint32_t e) {
                while (j < e && ref_key(j) < key) j = lds16(end_at + 2u * j);
            };

            // ---- the targets ----
            unsigned char* x0 = region + RankSmem::align16(sizeof(K) * nref);
            const uint32_t xbytes = (uint32_t)(reinterpret_cast<unsigned char*>(run_end) - x0);
            const uint32_t ntar = s_ntar;
            const bool ties = tk->tie_correction != 0;
            // no group's sum of the shares can leave the low word: plain adds, no carry
            const bool a32 = 2ull * nref * ntar <= 0xffffffffull;
            words_a = a32;
            const bool b32 = 3ull * s_maxrun * (s_maxrun + 1u) * ntar <= 0xffffffffull;
            // two bitmaps (cells hit, cells hit more than once): 64 cells per target, or so many that
            // a gene without repeats expects a quarter of a hit (2 n^2) and skips the second pass
            const uint32_t most = (xbytes / 2u) & ~15u;
            const unsigned long long wish = max(8ull * ntar, (unsigned long long)ntar * ntar / 4u) + 16u;
            const uint32_t half = (uint32_t)min((unsigned long long)most, wish & ~15ull), cells = half * 8u;
            const uint32_t hit_at = smem_addr(x0);
            if (ties)
                for (uint32_t i = tid; i < half / 8u; i += NT) reinterpret_cast<uint4*>(x0)[i] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
            auto load = [&](uint32_t at, K* key, uint2& g) {
                if (at < ntar) {
                    if constexpr (sizeof(K) == 4) {
                        const uint4 x = *reinterpret_cast<const uint4*>(dk + at);
                        key[0] = x.x; key[1] = x.y; key[2] = x.z; key[3] = x.w;
                    } else {
                        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(dk + at);
                        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(dk + at + 2);
                        key[0] = x.x; key[1] = x.y; key[2] = y.x; key[3] = y.y;
                    }
                    g = *reinterpret_cast<const uint2*>(dg + at);
                }
            };
            // the decoded targets, four neighbours per thread (groups beyond the last: 0), the next
            // four in flight; the first `skip` warps have other work
            auto stream = [&](int skip, auto f) {
                const uint32_t step = 4u * (uint32_t)(NT - 32 * skip);
                uint32_t i = 4u * (uint32_t)(tid - 32 * skip);
                K ka[4], kb[4];
                uint2 ga = make_uint2(0u, 0u), gb = make_uint2(0u, 0u);
                auto take = [&](K* key, const uint2& gp) {
                    uint32_t g[4] = {gp.x & 0xffffu, gp.x >> 16, gp.y & 0xffffu, gp.y >> 16};
                    const uint32_t left = ntar - i;
                    if (left < 4u) {
#pragma unroll
                        for (uint32_t k = 1; k < 4; ++k)
                            if (k >= left) { g[k] = 0u; key[k] = key[0]; }
                    }
                    f(key, g, i);
                };
                load(i, ka, ga);
                while (i < ntar) {  // (the two sets of registers take turns)
                    load(i + step, kb, gb);
                    take(ka, ga);
                    i += step;
                    if (i >= ntar) break;
                    load(i + step, ka, ga);
                    take(kb, gb);
                    i += step;
                }
            };
            uint32_t hits = 0, more = 0;  // entries in cells hit before, cells hit more than once
            const uint32_t a_at = smem_addr(a32s), nz_off = smem_addr(nz) - a_at, ng_off = smem_addr(ng) - a_at,
                           b_off = smem_addr(b32s) - a_at;
            const int pvw = pv_tk ? min(kPvWarps, (pv_tk->G + 30) / 32) : 0;
            if (warp < pvw) {
                pvalue_tiles(pv_tk, pv_c, &s_pvq, a.erfc_table);
            } else {
                // the four elements of a lane go through each stage together, so that their
                // dependent shared-memory reads overlap; a key that its bucket's first value
                // does not place walks on
                stream(pvw, [&](const K* key, const uint32_t* g, uint32_t i) {
                    K first[4];
                    uint32_t lo[4], hi[4], end[4], eq[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t b = bs_at + 4u * bmap.template at<VM>(key[k]);
                        lo[k] = lds(b - 4u);
                        hi[k] = lds(b);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        first[k] = ref_key(lo[k]);
                        end[k] = lds16(end_at + 2u * lo[k]);  // (lo = nref: readable, unused)
                    }
                    bool on = false;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const bool in = lo[k] < hi[k];
                        eq[k] = in && first[k] == key[k] ? end[k] - lo[k] : 0u;
                        if (in && first[k] < key[k]) lo[k] = end[k];
                        else hi[k] = 0u;
                        on |= lo[k] < hi[k];
                    }
                    if (on) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            if (lo[k] < hi[k]) {
                                walk(key[k], lo[k], hi[k]);
                                if (lo[k] < hi[k] && ref_key(lo[k]) == key[k]) eq[k] = lds16(end_at + 2u * lo[k]) - lo[k];
                            }
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t at = a_at + 4u * g[k], x = 2u * lo[k] + eq[k];
                        if (a32) {
                            if (g[k]) reds(at, x);
                        } else if (g[k]) {
                            acc_add<true>(&A[g[k]], x);
                        }
                        if (g[k]) reds(at + nz_off, 1u);
                        if (zh == ZH_MIX && g[k] && key[k] < k0) reds(at + ng_off, 1u);
                        if (ties && g[k] && eq[k]) {
                            const uint32_t y = 3u * eq[k] * (eq[k] + 1u);
                            if (b32) reds(at + b_off, y);
                            else acc_add<true>(&B[g[k]], y);
                        }
                    }
                    if (!ties) return;
                    uint32_t old[4], bit[4], at[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t cell = __umulhi(pair_hash(key[k], g[k]), cells);
                        bit[k] = 1u << (cell & 31u);
                        at[k] = hit_at + 4u * (cell >> 5);
                        old[k] = 0u;
                        if (g[k]) old[k] = ors(at[k], bit[k]);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (old[k] & bit[k]) {
                            ++hits;
                            more += !(ors(at[k] + half, bit[k]) & bit[k]);
                        }
                    }
                });
                if (pv_tk) pvalue_tiles(pv_tk, pv_c, &s_pvq, a.erfc_table);  // what is left of them
            }
            hits = __reduce_add_sync(0xffffffffu, hits);
            more = __reduce_add_sync(0xffffffffu, more);
            if (lane == 0 && hits) { atomicAdd(&s_hits, hits); atomicAdd(&s_cells, more); }
            __syncthreads();
            if (!ties) return;
            if (s_hits) {
                // distinct pairs to count: one per cell hit more than once and one per further
                // pair sharing it, of which n^2 / 2 cells are expected
                const float share = 0.5f * (float)ntar * (float)ntar / (float)cells;
                const float want = 1.1f * ((float)s_cells + fminf((float)s_hits, share)) + 64.0f;
                // a slot counts to 65,535; the elements counted are those of cells hit more than once
                const bool wide = s_hits + s_cells > 0xffffu;
                // The elements of cells hit more than once, each warp's to the front of its own part
                // of the slice (never ahead of what it has read), so that the lanes that count
                // below are all busy: one element in six of a screen's, too few in any warp.
                constexpr uint32_t W = NT / 32;
                const uint32_t seg = (ntar + 128u * W - 1u) / (128u * W) * 128u;
                const uint32_t s0 = min(ntar, (uint32_t)warp * seg), s1 = min(ntar, s0 + seg);
                uint32_t found = s0;
                {
                    K key[4] = {}, next[4] = {};
                    uint2 gp = make_uint2(0u, 0u), gn = make_uint2(0u, 0u);
                    const unsigned below = (1u << lane) - 1u;
                    load(s0 + 4u * lane, key, gp);
                    for (uint32_t t = s0; t < s1; t += 128u) {
                        const uint32_t i = t + 4u * lane;
                        if (t + 128u < s1) load(i + 128u, next, gn);
                        const uint32_t g[4] = {gp.x & 0xffffu, gp.x >> 16, gp.y & 0xffffu, gp.y >> 16};
                        uint32_t cell[4], w[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            cell[k] = __umulhi(pair_hash(key[k], g[k]), cells);
                            w[k] = lds(hit_at + half + 4u * (cell[k] >> 5));
                        }
                        __syncwarp();
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const bool on = i + k < ntar && ((w[k] >> (cell[k] & 31u)) & 1u);
                            const unsigned m = __ballot_sync(0xffffffffu, on);
                            if (on) {
                                const uint32_t o = found + __popc(m & below);
                                dk[o] = key[k];
                                dg[o] = (GT)g[k];
                            }
                            found += __popc(m);
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k) key[k] = next[k];
                        gp = gn;
                    }
                }
                // the table in the place of the bitmaps, at most three quarters full
                PairTable table{reinterpret_cast<unsigned long long*>(x0), 0u};
                const uint32_t room = (xbytes / 16u) * 2u;
                uint32_t parts = 1;
                while (want > 0.75f * (float)room * (float)parts && parts < 64u) parts *= 2u;
                table.n = min(room, ((uint32_t)(2.0f * want) / parts + 32u) & ~1u);
                for (uint32_t q = 0; q < parts; ++q) {
                    __syncthreads();
                    for (uint32_t p = tid; p < table.n / 2u; p += NT) reinterpret_cast<uint4*>(table.slot)[p] = make_uint4(0u, 0u, 0u, 0u);
                    __syncthreads();
                    for (uint32_t i = s0 + lane; i < found; i += 32u) {
                        const K key = dk[i];
                        const uint32_t g = dg[i], h = pair_hash(key, g);
                        if (((h >> 5) & (parts - 1u)) == q && !pair_count<K>(table, key, g, i, h * 0x9e3779b1u, dk, wide))
                            s_bad = 1u;
                    }
                    __syncthreads();
                    if (s_bad) return;
                    // pairs counted more than once
                    for (uint32_t p = tid; p < table.n; p += NT) {
                        const unsigned long long cur = table.slot[p];
                        const unsigned long long s = cur & 0xffffull;
                        const uint32_t g = ((uint32_t)cur >> 16);
                        if (s < 2ull || g >= (uint32_t)G) continue;
                        const K key = slot_key<K>(cur, dk);
                        const uint32_t b = bmap.template at<VM>(key), e = bs[b];
                        uint32_t j = bucket_start(b);
                        walk(key, j, e);
                        const unsigned long long equal = j < e && ref_key(j) == key ? run_end[j] - j : 0u;
                        acc_add<true>(&B[g], 3ull * equal * (s * s - s) + s * s * s - s);
                    }
                }
            }
        };
        if (BucketMap<V>::signed_range(kmin, kmax)) gene(std::true_type{});
        else gene(std::false_type{});
        if (tid == NT - 1) fetch_gene();
        // pending p-values not taken beside the targets (a gene that was left has none)
        if (pv_tk) pvalue_tiles(pv_tk, pv_c, &s_pvq, a.erfc_table);
        tref = warp_sum_u64(tref);
        if (lane == 0 && tref) atomicAdd(&s_tref, tref);
        if (tid == 0) { nz[0] = s_nref; ng[0] = s_neg; }
        __syncthreads();
        // the decoded targets are dead: drop their lines from L2 instead of writing them back
        l2_discard<NT>(dk, (size_t)s_ntar * sizeof(K));
        l2_discard<NT>(dg, (size_t)s_ntar * sizeof(GT));
        const bool bad = s_bad != 0u;
        if (tid == NT - 1) fetch_column();
        if (!bad)
            for (int g = 1 + tid; g < G; g += NT)
                finalize_target(tk, c, G, zh, g, words_a ? (unsigned long long)a32s[g] : A[g], B[g] + b32s[g],
                                nz, ng, s_tref);
        if (tid == 0) {
            if (bad) {
                const int k = atomicAdd(a.n_left, 1);
                a.left[k] = c;
                if (a.left_task) a.left_task[k] = (uint16_t)ti;
            }
            s_pv_gene = (a.erfc_table && !bad) ? c : -1;
            s_pv_task = ti;
            s_pvq = 0u;
        }
        __syncthreads();
    }
}

}  // namespace hpdex
