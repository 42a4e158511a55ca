// group_mean.cuh -- per (gene, group) means over a CSC matrix (sm_103a).
//
// Restates hpdex::group_mean_core (AI4Cell/hpdex src/cpp/mannwhitneyu.cpp:1118-1192): for
// every gene and group, the sum of the finite explicit values of rows in the group divided
// by group_rows[g] - invalid[g] (include_zeros; implicit zeros count, non-finite entries
// do not) or by valid[g] (explicit values only); a zero denominator gives 0. Output is
// flat [gene * G + g] like the reference. One CTA per gene.
//
// A double atomic add in shared memory is a compare-and-swap loop, which
// on a gene's random groups retries for every lane that shares a word, while a 32-bit integer
// add is a single native operation. So a gene's values are added as fixed-point integers of 64 or 96 bits
// (two or three 32-bit words with the carry taken from the returned old value), scaled by a
// power of two that its key range and entry count choose so that the largest sum does not
// overflow. Such sums are exact and do not depend on the order of the atomics; one rounding turns
// them into doubles. They hold every bit of the gene's values unless the lowest bit of some value lies
// more than 94 bits, less those of the entry count, below the top of the largest (doubles: a
// value below 2^-25 of the largest in a gene of 100,000 entries; float32: 2^-54). A value that would
// lose a bit makes the CTA repeat the gene with double atomics, whose sums round once per
// addition and depend on their order; the same holds for more groups than shared memory has room
// for. (300 genes of 200,000 float32 values over 30 decades: 1.36 ms, double atomics at once 1.30. A test
// that ends the first pass at such a value gave 1.11, but cost the genes of three words that
// lose none up to 9%.)
#pragma once
#include <cstdint>
#include <type_traits>

#include "common.cuh"

namespace hpdex {

struct MeanArgs {
    const void* data;
    const int32_t* rows;
    const int64_t* indptr;
    const unsigned long long* col_kmin;  // key range of the finite nonzero values and flags of each
    const unsigned long long* col_kmax;  //   column, as in RankTask
    const uint32_t* col_flags;
    int64_t n_rows;
    int32_t n_cols;
    int32_t G;
    const int32_t* gid;            // group_mean_kernel
    const uint16_t* gid16;         // group_mean_fixed_kernel (all ones: in no group)
    const unsigned int* group_rows;
    int32_t include_zeros;
    double* out;                   // [n_cols * G]
    unsigned char* acc_global;     // per CTA 16*G bytes (group_mean_kernel)
};

// Rows of each group (cnt zeroed before) and, for GT = uint16_t, the group ids in 16 bits.
// SMEM: counted per block in shared memory first (G counters fit).
template <bool SMEM>
__global__ void group_rows_kernel(const int32_t* gid, long long n_rows, int32_t G, unsigned int* cnt,
                                  uint16_t* gid16) {
    extern __shared__ unsigned int grp_cnt_s[];
    if constexpr (SMEM) {
        for (int g = threadIdx.x; g < G; g += blockDim.x) grp_cnt_s[g] = 0u;
        __syncthreads();
    }
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += stride) {
        const int32_t g = gid[r];
        const bool in = g >= 0 && g < G;
        if (in) atomicAdd(SMEM ? &grp_cnt_s[g] : &cnt[g], 1u);
        if (gid16) gid16[r] = in ? (uint16_t)g : (uint16_t)0xffff;
    }
    if constexpr (SMEM) {
        __syncthreads();
        for (int g = threadIdx.x; g < G; g += blockDim.x)
            if (grp_cnt_s[g]) atomicAdd(&cnt[g], grp_cnt_s[g]);
    }
}

__device__ __forceinline__ double mean_of(double sum, const MeanArgs& a, int g, uint32_t valid,
                                          uint32_t invalid) {
    const long long denom = a.include_zeros ? (long long)a.group_rows[g] - (long long)invalid
                                            : (long long)valid;
    return denom > 0 ? __ddiv_rn(sum, (double)denom) : 0.0;
}

// Any number of groups: double atomics on accumulators in global memory.
template <class V, int NT>
__global__ void __launch_bounds__(NT) group_mean_kernel(const MeanArgs a) {
    const int G = a.G, tid = threadIdx.x;
    double* sum = reinterpret_cast<double*>(a.acc_global + (size_t)blockIdx.x * 16 * G);
    uint32_t* valid = reinterpret_cast<uint32_t*>(sum + G);
    uint32_t* invalid = valid + G;
    const V* data = reinterpret_cast<const V*>(a.data);

    for (int c = blockIdx.x; c < a.n_cols; c += gridDim.x) {
        for (int g = tid; g < G; g += NT) { sum[g] = 0.0; valid[g] = 0u; invalid[g] = 0u; }
        __syncthreads();
        const long long p0 = a.indptr[c], p1 = a.indptr[c + 1];
        for (long long p = p0 + tid; p < p1; p += NT) {
            const long long r = a.rows[p];
            if (r < 0 || r >= a.n_rows) continue;
            const int g = a.gid[r];
            if (g < 0 || g >= G) continue;
            const V v = data[p];
            if (Val<V>::finite(v)) {
                atomicAdd(&sum[g], Val<V>::to_double(v));
                atomicAdd(&valid[g], 1u);
            } else {
                atomicAdd(&invalid[g], 1u);
            }
        }
        __syncthreads();
        for (int g = tid; g < G; g += NT)
            a.out[(size_t)c * G + g] = mean_of(sum[g], a, g, valid[g], invalid[g]);
        __syncthreads();
    }
}

// A finite value as (-1)^neg * m * 2^e with an integer m: float32 values from their bits, the
// other types from the integer or double that the reference adds.
struct FixedValue {
    unsigned long long m;
    int e;
    bool neg;
};
template <class V>
__device__ __forceinline__ FixedValue fixed_value(V v) {
    FixedValue f;
    if constexpr (std::is_same_v<V, float>) {
        const uint32_t b = __float_as_uint(v);
        const int x = (int)((b >> 23) & 0xffu);
        f.m = (b & 0x7fffffu) | (x ? 0x800000u : 0u);
        f.e = (x ? x : 1) - 150;
        f.neg = (b >> 31) != 0u;
    } else if constexpr (sizeof(V) == 8) {  // double, or a 64-bit integer added as its double
        const unsigned long long b = (unsigned long long)__double_as_longlong(Val<V>::to_double(v));
        const int x = (int)((b >> 52) & 0x7ffull);
        f.m = (b & 0xfffffffffffffull) | (x ? 1ull << 52 : 0ull);
        f.e = (x ? x : 1) - 1075;
        f.neg = (b >> 63) != 0ull;
    } else {
        const long long x = (long long)v;
        f.neg = x < 0;
        f.m = (unsigned long long)(f.neg ? -x : x);
        f.e = 0;
    }
    return f;
}

// The scale of a gene: values are multiples of 2^-scale, sums stay below 2^62 (two words) or
// 2^94 (three words).
struct FixedScale {
    int scale;
    bool wide;   // three words
    bool word;   // every value is one unsigned word (fixed_word)
};
template <class V>
__device__ __forceinline__ FixedScale fixed_scale(unsigned long long kmin, unsigned long long kmax,
                                                  uint32_t flags, long long nnz) {
    using K = typename Val<V>::Key;
    constexpr bool kFloat = std::is_same_v<V, float> || std::is_same_v<V, double>;
    FixedScale s{0, false, !kFloat};
    if ((K)kmin > (K)kmax) return s;  // no finite nonzero value
    auto exponent = [](double x) {    // |x| < 2^exponent (float32 and larger magnitudes are normal)
        const int e = (int)(((unsigned long long)__double_as_longlong(x) >> 52) & 0x7ffull);
        return e ? e - 1022 : -1022;
    };
    const double lo = Val<V>::from_key((K)kmin), hi = Val<V>::from_key((K)kmax);
    const int top = max(exponent(lo), exponent(hi));
    const int cnt = 64 - __clzll(nnz);
    int unit = 0;  // every value is a multiple of 2^unit (integers: 2^0)
    if (kFloat && (flags & 2u)) {
        constexpr int mant = std::is_same_v<V, float> ? 24 : 53, least = std::is_same_v<V, float> ? -149 : -1074;
        unit = lo > 0.0 ? max(exponent(lo) - mant, least) : top + cnt - 94;
    }
    if (top - unit + cnt > 94) unit = top + cnt - 94;
    s.scale = -unit;
    s.wide = top - unit + cnt > 62;
    s.word = !std::is_same_v<V, double> && lo >= 0.0 && top - unit <= 32 && s.scale >= -126 && s.scale <= 127;
    return s;
}

// The value times 2^scale of a gene whose values are all words: one multiplication and one
// conversion for float32 (both exact), the value itself for integers.
template <class V>
__device__ __forceinline__ uint32_t fixed_word(V v, float unit) {
    if constexpr (std::is_same_v<V, float>) return __float2uint_rn(v * unit);
    else return (uint32_t)v;
}
// Adds a word to the 64-bit sum `i` (two words, `n` apart).
__device__ __forceinline__ void fixed_add_word(uint32_t* w, int n, uint32_t i, uint32_t x) {
    const uint32_t old = atomicAdd(&w[i], x);
    if (old + x < old) atomicAdd(&w[n + i], 1u);
}

// Adds a value to accumulator `i` of the word arrays w (stride `n` words between them); false
// when bits would be lost.
template <bool WIDE>
__device__ __forceinline__ bool fixed_add(uint32_t* w, int n, int i, const FixedValue& f, int scale) {
    const int sh = f.e + scale;
    unsigned long long lo, hi = 0ull;
    if (sh >= 0) {
        if constexpr (WIDE) {
            lo = sh < 64 ? f.m << sh : 0ull;
            hi = sh == 0 ? 0ull : sh < 64 ? f.m >> (64 - sh) : f.m << (sh - 64);
        } else {
            lo = f.m << sh;
        }
    } else {
        lo = sh > -64 ? f.m >> -sh : 0ull;
        if (sh <= -64 ? f.m != 0ull : (lo << -sh) != f.m) return false;
    }
    if (f.neg) {
        lo = 0ull - lo;
        hi = ~hi + (lo == 0ull ? 1ull : 0ull);
    }
    const uint32_t a0 = (uint32_t)lo, a1 = (uint32_t)(lo >> 32);
    uint32_t c = 0u;
    if (a0) {
        const uint32_t old = atomicAdd(&w[i], a0);
        c = (uint32_t)(old + a0 < old);
    }
    const uint32_t b1 = a1 + c;
    if constexpr (WIDE) {
        uint32_t c2 = (uint32_t)(b1 < c);
        if (b1) {
            const uint32_t old = atomicAdd(&w[n + i], b1);
            c2 += (uint32_t)(old + b1 < old);
        }
        const uint32_t b2 = (uint32_t)hi + c2;
        if (b2) atomicAdd(&w[2 * n + i], b2);
    } else {
        if (b1) atomicAdd(&w[n + i], b1);
    }
    return true;
}

// The double nearest to the 96-bit two's complement integer (hi, lo) * 2^-scale.
__device__ __forceinline__ double fixed_double(unsigned long long lo, int32_t hi, int scale) {
    const bool neg = hi < 0;
    uint32_t h = (uint32_t)hi;
    if (neg) {
        lo = 0ull - lo;
        h = ~h + (lo == 0ull ? 1u : 0u);
    }
    int up = 0;
    if (h) {  // the top 64 bits, the rest of them as a sticky bit below the rounding position
        up = 32 - __clz((int)h);
        const bool rest = (lo & ((1ull << up) - 1ull)) != 0ull;
        lo = (lo >> up) | ((unsigned long long)h << (64 - up)) | (rest ? 1ull : 0ull);
    }
    const double d = scalbn(__ull2double_rn(lo), up - scale);
    return neg ? -d : d;
}

// Up to 65,534 groups whose accumulators fit in shared memory (three words of sums per group,
// then valid / invalid): fixed-point sums as above, one CTA per gene. Four entries per thread are
// loaded while the previous four are gathered and added. Bound by instruction issue and the shared
// atomics: the screen (1.47e8 entries, 501 groups) 5.94 ms with double atomics, 0.47 ms with
// the two-word sums for every gene, 0.37 ms (3.2 TB/s) with genes of one-word values taking the
// short form (fixed_word); integer counts (3.5e7 entries, 50 groups) 3.51, 0.13 and 0.083 ms.
// Several accumulator sets, taken by lane to keep lanes of one group apart, gained nothing at 50
// groups (2, 4 or 8 sets) and lost time at 501.
template <class V, int NT>
__global__ void __launch_bounds__(NT, 3) group_mean_fixed_kernel(const MeanArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_lost;
    const int G = a.G, tid = threadIdx.x, c = blockIdx.x;
    uint32_t* w = reinterpret_cast<uint32_t*>(smem);
    double* sum = reinterpret_cast<double*>(smem);
    uint32_t* valid = w + 3 * G;
    uint32_t* invalid = valid + G;
    const long long p0 = a.indptr[c];
    const uint32_t nnz = (uint32_t)(a.indptr[c + 1] - p0), nrows = (uint32_t)a.n_rows;
    const int32_t* rows = a.rows + p0;
    const V* data = reinterpret_cast<const V*>(a.data) + p0;
    const FixedScale fs = fixed_scale<V>(a.col_kmin[c], a.col_kmax[c], a.col_flags[c], nnz);
    const int words = fs.wide ? 3 : 2;
    for (int i = tid; i < words * G; i += NT) w[i] = 0u;
    for (int i = tid; i < 2 * G; i += NT) valid[i] = 0u;
    if (tid == 0) s_lost = 0;
    __syncthreads();

    // every finite value of a row in a group goes to `add`; `count`: valid / invalid counts too
    auto pass = [&](auto add, bool count) {
        int32_t r[4];
        V v[4];
        auto load = [&](uint32_t t, int32_t* rr, V* vv) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t i = t + (uint32_t)k * NT;
                rr[k] = i < nnz ? __ldcs(rows + i) : -1;
                vv[k] = i < nnz ? data[i] : V(0);
            }
        };
        load(tid, r, v);
        for (uint32_t t = tid; t < nnz; t += 4u * NT) {
            int32_t rn[4];
            V vn[4];
            uint32_t g[4];
            load(t + 4u * NT, rn, vn);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                g[k] = (uint32_t)r[k] < nrows ? (uint32_t)__ldg(a.gid16 + r[k]) : 0xffffu;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (g[k] != 0xffffu) {
                    if (Val<V>::finite(v[k])) {
                        add(g[k], v[k]);
                        if (count && !a.include_zeros) atomicAdd(&valid[g[k]], 1u);
                    } else if (count) {
                        atomicAdd(&invalid[g[k]], 1u);
                    }
                }
                r[k] = rn[k];
                v[k] = vn[k];
            }
        }
    };
    bool lost = false;
    const float unit = __int_as_float((uint32_t)(fs.scale + 127) << 23);  // 2^scale (fs.word)
    if (fs.word)
        pass([&](uint32_t g, V v) { fixed_add_word(w, G, g, fixed_word<V>(v, unit)); }, true);
    else if (fs.wide)
        pass([&](uint32_t g, V v) { lost |= !fixed_add<true>(w, G, (int)g, fixed_value<V>(v), fs.scale); }, true);
    else
        pass([&](uint32_t g, V v) { lost |= !fixed_add<false>(w, G, (int)g, fixed_value<V>(v), fs.scale); }, true);
    if (lost) s_lost = 1;
    __syncthreads();
    if (s_lost) {
        for (int g = tid; g < G; g += NT) sum[g] = 0.0;
        __syncthreads();
        pass([&](uint32_t g, V v) { atomicAdd(&sum[g], Val<V>::to_double(v)); }, false);
        __syncthreads();
    }
    for (int g = tid; g < G; g += NT) {
        double s;
        if (s_lost) {
            s = sum[g];
        } else {
            const unsigned long long lo = (unsigned long long)w[g] | ((unsigned long long)w[G + g] << 32);
            const int32_t hi = fs.wide ? (int32_t)w[2 * G + g] : ((int32_t)w[G + g] >> 31);
            s = fixed_double(lo, hi, fs.scale);
        }
        a.out[(size_t)c * G + g] = mean_of(s, a, g, valid[g], invalid[g]);
    }
}

}  // namespace hpdex
