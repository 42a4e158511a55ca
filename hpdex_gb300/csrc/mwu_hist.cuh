// mwu_hist.cuh -- integer-count genes ranked from (value, group) counters, several CTAs per SM (sm_103a).
//
// The histogram path of mwu_rank_kernel (mwu_rank.cuh) in a kernel of its own: the same counters,
// prefix and per-group sums. Inside that kernel a gene has an SM to itself, and its phases (clear,
// count, scan, groups, finalize) leave it idle at every barrier and load: 17 us a gene of 17,700
// entries, of which the counting is 6. The counters of a UMI gene are small (50 groups x 30 values:
// 6 KB), so here an SM holds four CTAs of 384 threads, each with a gene, and one's barriers
// are another's work; the p-values follow at once, without the pending tiles of the one-CTA
// kernels. Genes that are not small integers or span too many values are listed for
// mwu_rank_kernel, launched behind this one.
//
// Bound by the latency of a gene's phases and of its longest genes. Integer counts (50,000 x 2,000,
// 49 targets): 219 us in mwu_rank_kernel, 120 us here (2.4 TB/s); 512 threads x 4 / x 3 128 us,
// 256 x 6 165-185 us. Genes with values above the first range (285 at 50 groups) left to
// mwu_rank_kernel took 36 us behind it, a second pass over their columns 35 us; most hold fewer
// than 256 such elements, which are resolved pairwise.
#pragma once
#include "mwu_rank.cuh"

namespace hpdex {

struct HistArgs {
    const RankTask* tasks;
    const int32_t* order;        // genes in processing order [n_order]
    const uint16_t* order_task;  // task of each entry of `order` (null: all task 0)
    int32_t n_order;
    int32_t* queue;              // work counter
    int32_t G;                   // layout G: the largest task G of the launch
    int32_t words;               // counters per CTA
    const double* erfc_table;    // non-null: p-values too, as in RankArgs
    int32_t* left;               // genes (and tasks) left to mwu_rank_kernel, and how many
    uint16_t* left_task;
    int32_t* n_left;
};

constexpr int kHistThreads = 384;
constexpr int kHistCTAs = 4;
constexpr int kHistRanges = 8;  // ranges of values a gene may take
constexpr int kHistTail = 256;  // elements above the first range that are resolved pairwise instead

// Shared memory: sums and counts (24 bytes per group), then the counters.
__host__ __device__ inline size_t hist_acc_bytes(int G) { return RankSmem::align16((size_t)G * 24); }

template <class V, int NT, int CTAS>
__global__ void __launch_bounds__(NT, CTAS) mwu_hist_kernel(const HistArgs a) {
    using K = typename Val<V>::Key;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_gene, s_task;
    __shared__ long long s_p0, s_p1;
    __shared__ unsigned long long s_kmin, s_kmax, s_tref;
    __shared__ uint32_t s_flags;
    __shared__ uint32_t s_ws[32];
    __shared__ uint32_t s_tail[kHistTail];  // elements above the first range: value << 16 | group
    __shared__ uint32_t s_ntail, s_tailref, s_tailneg;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int GL = a.G;
    unsigned long long* A = reinterpret_cast<unsigned long long*>(smem);
    unsigned long long* B = A + GL;
    uint32_t* nz = reinterpret_cast<uint32_t*>(B + GL);
    uint32_t* ng = nz + GL;
    uint32_t* hc = reinterpret_cast<uint32_t*>(smem + hist_acc_bytes(GL));

    for (;;) {
        if (tid == 0) {
            const int gi = atomicAdd(a.queue, 1);
            s_gene = -1;
            if (gi < a.n_order) {
                const int c = a.order[gi], ti = a.order_task ? (int)a.order_task[gi] : 0;
                const RankTask* t = a.tasks + ti;
                s_gene = c;
                s_task = ti;
                s_p0 = t->indptr[c];
                s_p1 = t->indptr[c + 1];
                s_kmin = t->col_kmin[c];
                s_kmax = t->col_kmax[c];
                s_flags = t->col_has_zero[c];
                s_tref = 0ull;
                s_ntail = 0u;
                s_tailref = 0u;
                s_tailneg = 0u;
            }
        }
        __syncthreads();
        const int c = s_gene;
        if (c < 0) break;
        const RankTask* tk = a.tasks + s_task;
        const int G = tk->G, zh = tk->zero_handling;
        const uint16_t* gidp = reinterpret_cast<const uint16_t*>(tk->group_of_row);
        const uint32_t nrows = (uint32_t)tk->n_rows, nraw = (uint32_t)(s_p1 - s_p0);
        const int32_t* rows = tk->rows + s_p0;
        const V* data = reinterpret_cast<const V*>(tk->data) + s_p0;
        K kmin = (K)s_kmin, kmax = (K)s_kmax;
        if (zh == ZH_NONE && (s_flags & 1u)) {
            const K kz = Val<V>::key(V(0));
            kmin = kz < kmin ? kz : kmin;
            kmax = kz > kmax ? kz : kmax;
        }
        // the gene's values up to W, whose counters fit; the elements above them (a UMI gene's few
        // large counts) pairwise, or where they are many in further ranges, for each of which the
        // column is read again (from L2)
        int hV = 0, hVp = 0;
        long long lo = 0;
        bool fits = false;
        const int W = min((a.words - 4) / G, 8 * NT - 8) & ~3;
        if (!(s_flags & 2u) && kmin <= kmax && W > 0) {
            lo = (long long)Val<V>::from_key(kmin);
            fits = hist_choice(lo, (long long)Val<V>::from_key(kmax), G, nraw, 1ll << 40, &hV, &hVp) &&
                   hV <= kHistRanges * W;
        }
        if (!fits) {
            if (tid == 0) {
                const int k = atomicAdd(a.n_left, 1);
                a.left[k] = c;
                if (a.left_task) a.left_task[k] = (uint16_t)s_task;
            }
            __syncthreads();  // (the gene's fields are read)
            continue;
        }
        unsigned long long tref = 0ull;
        uint32_t below = 0, negref = 0;  // reference elements in the ranges before, and below 0
        for (int base = 0; base < hV; base += W) {
        const int Vr = min(W, hV - base), Vp = (Vr + 3) & ~3;
        const int words = (int)hist_words(Vp, G);
        for (int i = 4 * tid; i < words; i += 4 * NT) *reinterpret_cast<uint4*>(hc + i) = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();

        // ---- one streaming pass: each stored element increments its (value, group) counter ----
        {
            int32_t r[4];
            V v[4];
            auto load = [&](uint32_t t, int32_t* rr, V* vv) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t e = t + (uint32_t)k * NT;
                    rr[k] = e < nraw ? __ldcs(rows + e) : -1;
                    vv[k] = e < nraw ? ld_stream(data + e) : V(0);
                }
            };
            load(tid, r, v);
            for (uint32_t t = tid; t < nraw; t += 4u * NT) {
                int32_t rn[4];
                V vn[4];
                uint32_t g[4];
                load(t + 4u * NT, rn, vn);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    g[k] = (uint32_t)r[k] < nrows ? (uint32_t)__ldg(gidp + r[k]) : 0xffffu;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t bin = hist_bin<V>(v[k], lo + base);
                    if (g[k] != 0xffffu && Val<V>::finite(v[k]) && (zh == ZH_NONE || !Val<V>::zero(v[k]))) {
                        if (bin < (uint32_t)Vr) {
                            red_add<true>(&hc[(g[k] ? 4u + g[k] * (uint32_t)Vp : 0u) + bin], 1u);
                        } else if (base == 0) {
                            const uint32_t q = atomicAdd(&s_ntail, 1u);
                            if (q < (uint32_t)kHistTail) s_tail[q] = bin << 16 | g[k];
                        }
                    }
                    r[k] = rn[k];
                    v[k] = vn[k];
                }
            }
        }
        __syncthreads();
        block_scan1<NT>(hc, Vr, s_ws);  // hc[v] = reference elements below v, hc[Vr] = all of them

        // ---- one warp per target group: its row against the reference's prefix counts ----
        for (int g = 1 + warp; g < G; g += NT / 32) {
            const uint32_t* row = hc + 4 + (size_t)g * Vp;
            unsigned long long sa = 0, sb = 0;
            uint32_t snz = 0, sng = 0;
            for (int v = lane; v < Vr; v += 32) {
                const uint32_t sv = row[v];
                if (sv) {
                    const uint32_t R = hc[v], rv = hc[v + 1] - R;
                    sa += (unsigned long long)sv * (2ull * (below + R) + rv);
                    sb += tie_delta(rv, sv);
                    snz += sv;
                    if (lo + base + v < 0) sng += sv;
                }
            }
            sa = warp_sum_u64(sa);
            sb = warp_sum_u64(sb);
            snz = __reduce_add_sync(0xffffffffu, snz);
            sng = __reduce_add_sync(0xffffffffu, sng);
            if (lane == 0) {
                if (base == 0) { A[g] = sa; B[g] = sb; nz[g] = snz; ng[g] = sng; }
                else { A[g] += sa; B[g] += sb; nz[g] += snz; ng[g] += sng; }
            }
        }
        for (int v = tid; v < Vr; v += NT) {
            const unsigned long long rv = hc[v + 1] - hc[v];
            tref += rv * rv * rv - rv;
        }
        if (lo + base < 0) negref += hc[(int)min(-(lo + base), (long long)Vr)];
        below += hc[Vr];
        __syncthreads();
        if (base == 0 && hV > W && s_ntail <= (uint32_t)kHistTail) {
            // few elements above the first range: each counts, over the list, the reference
            // elements below and equal to it and its own repeats, and adds its share
            const uint32_t n = s_ntail;
            uint32_t nref = 0, nneg = 0;
            for (uint32_t i = tid; i < n; i += NT) {
                const uint32_t w = s_tail[i], v = w >> 16, g = w & 0xffffu;
                uint32_t lt = 0, eq = 0, same = 0;
                for (uint32_t j = 0; j < n; ++j) {
                    const uint32_t x = s_tail[j];
                    same += x == w;
                    lt += (x & 0xffffu) == 0u && (x >> 16) < v;
                    eq += x == (v << 16);
                }
                if (g) {
                    acc_add<true>(&A[g], 2ull * (below + lt) + eq);
                    acc_add<true>(&B[g], 3ull * eq * eq + 3ull * eq * same + (unsigned long long)same * same - 1ull);
                    red_add<true>(&nz[g], 1u);
                    if (lo + v < 0) red_add<true>(&ng[g], 1u);
                } else {
                    tref += (unsigned long long)eq * eq - 1ull;
                    ++nref;
                    nneg += lo + v < 0;
                }
            }
            if (nref) atomicAdd(&s_tailref, nref);
            if (nneg) atomicAdd(&s_tailneg, nneg);
            __syncthreads();
            below += s_tailref;
            negref += s_tailneg;
            break;
        }
        }
        tref = warp_sum_u64(tref);
        if (lane == 0 && tref) atomicAdd(&s_tref, tref);
        if (tid == 0) { nz[0] = below; ng[0] = negref; }
        __syncthreads();

        // ---- U1, tie sum and p-value per target, by the thread that owns it ----
        for (int g = 1 + tid; g < G; g += NT) finalize_target(tk, c, G, zh, g, A[g], B[g], nz, ng, s_tref);
        if (a.erfc_table) {
            if (zh == ZH_NONE) __syncthreads();  // (the sample sizes of the gene, written by one thread)
            for (uint32_t q = warp; 32u * q + 1u < (uint32_t)G; q += NT / 32) pvalue_tile(tk, c, q, a.erfc_table);
        }
        __syncthreads();
    }
}

}  // namespace hpdex
