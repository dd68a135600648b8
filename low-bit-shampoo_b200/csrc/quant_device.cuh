// Device-side pieces of the blockwise quantizer that more than one kernel needs: the per-CTA
// codebook tables (exact decision thresholds + packed lookup table), the exact division and the
// generic per-lane routine.  Included by the stand-alone quantize kernels and by the GEMM whose
// epilogue writes 4-bit state.
#pragma once
#include "qt_common.cuh"
#include <math_constants.h>

namespace qt {

static constexpr int kLutMaxBits = 11;        // finest grid of the 16-entry table: 2048 cells over q in [-1, 1)

// ------------------------------------------------------------------------------------
// Codebook tables, built per CTA in shared memory.
// ------------------------------------------------------------------------------------
// 256-entry codebooks: cells of q are taken from its bit pattern - sign, exponent and the top six mantissa
// bits - so that they are narrow where codebooks are dense (near zero) and 1.6 % wide at |q| = 1: the squared-linear and
// the dynamic codebook have at most one threshold per cell.  Twenty octaves below 1, one cell for everything smaller.
static constexpr int kCellShift8 = 17;                       // mantissa bits inside a cell
static constexpr int kCellBase8 = ((127 - 20) << 6) - 1;     // (bits(|q|) >> 17) of the cell below 2^-20
static constexpr int kCells8 = 20 * 64 + 2;                  // cells per sign: smaller, 2^-20 .. 1, and 1 itself
template <int NC>
struct CodeTables {
    float raw[NC];
    float sorted[NC];
    float thr[NC];            // thr[j], j < NC-1: smallest q that rounds up from sorted[j]; thr[NC-1] = +inf
    unsigned char perm[NC];   // sorted position -> caller's code index
    float cmin, cmax;
    int perm_identity;
    int need_clamp;
    int lut_bad;
    int tiny_thr;             // some decision threshold has |t| < 2^-50: quotients must be exact even when tiny
    int thr_cell[NC];         // 256 entries: cell of each threshold; 16 entries: bit pattern of 3 + threshold
    // 16-entry codebooks: one word per cell of u = x / absmax + 3 (in [2, 4], so that its mantissa is linear in the
    // quotient and its upper bits number the cells).  bits(u) + word holds the code in its top byte and, in the
    // lower 24 bits, the distance of u above the cell's threshold plus four: see code_word().
    int lut_shift;            // byte offset of a cell's word: (bits(u) >> lut_shift) & lut_mask
    unsigned lut_mask;
    unsigned lut[NC == 16 ? (1 << kLutMaxBits) + 1 : 1];
    // 256-entry codebooks: one word per [sign][cell]: bits 31..14 = low mantissa bits from which the code is one
    // higher (q >= 0) or no longer one higher (q < 0); bit 8 = more than one threshold in the cell (take the search);
    // bits 7..0 = number of thresholds in lower cells.  The comparison is exact: cell and low bits are the whole of |q|.
    unsigned lut8[NC == 256 ? 2 * kCells8 : 1];
};

// Cell of |q| given its bit pattern without the sign, clamped to [0, kCells8 - 1] for |q| <= 1.
__device__ __forceinline__ int cell8_of(unsigned mag) { return max((int)(mag >> kCellShift8) - kCellBase8, 0); }

__device__ __forceinline__ long long float_key(float f) {
    int i = __float_as_int(f);
    return (long long)(i >= 0 ? i : (i ^ 0x7fffffff));
}
__device__ __forceinline__ float key_float(long long k) {
    int i = (int)k;
    return __int_as_float(i >= 0 ? i : (i ^ 0x7fffffff));
}
template <int NC>
__device__ void build_tables(CodeTables<NC> &t, const float *__restrict__ code) {
    const int tid = threadIdx.x;
    for (int i = tid; i < NC; i += blockDim.x) t.raw[i] = code[i];
    if (tid == 0) { t.lut_bad = 0; t.tiny_thr = 0; }
    __syncthreads();
    // The reference sorts a codebook that is not ascending (functional.py:561-565); an ascending one keeps its order.
    bool asc = true;
    for (int i = tid; i + 1 < NC; i += blockDim.x) asc = asc && (t.raw[i] <= t.raw[i + 1]);
    const int sorted = __syncthreads_and(asc);
    for (int i = tid; i < NC; i += blockDim.x) {
        const float v = t.raw[i];
        int rank = i;
        if (!sorted) {                                        // stable rank sort
            rank = 0;
            for (int j = 0; j < NC; ++j) {
                float w = t.raw[j];
                rank += (w < v) || (w == v && j < i);
            }
        }
        t.sorted[rank] = v;
        t.perm[rank] = (unsigned char)i;
    }
    __syncthreads();
    bool ident = true;
    for (int j = tid; j < NC; j += blockDim.x) {
        ident = ident && t.perm[j] == j;
        if (j == NC - 1) { t.thr[j] = CUDART_INF_F; continue; }
        const float lo = t.sorted[j], hi = t.sorted[j + 1];
        // predicate P(q) = |q - lo| > |hi - q| is false at lo and monotone in q
        long long a = float_key(lo), b = float_key(hi);
        if (!(fabsf(hi - lo) > 0.0f)) { t.thr[j] = hi; continue; }
        auto up = [&](long long k) { const float q = key_float(k); return fabsf(q - lo) > fabsf(hi - q); };
        // the threshold is within a few ulp of the midpoint: bisect there first (5 steps instead of 31)
        const long long mid = float_key(0.5f * lo + 0.5f * hi);
        if (mid - 16 > a && !up(mid - 16)) a = mid - 16;
        if (mid + 16 < b && up(mid + 16)) b = mid + 16;
        for (int it = 0; it < 64 && b - a > 1; ++it) {
            const long long m = a + ((b - a) >> 1);
            if (up(m)) b = m; else a = m;
        }
        t.thr[j] = key_float(b);
        if (fabsf(t.thr[j]) < 8.8817842e-16f) t.tiny_thr = 1;             // 2^-50
    }
    const int all_ident = __syncthreads_and(ident);           // also: thresholds are visible
    if (tid == 0) {
        t.perm_identity = all_ident;
        t.cmin = t.sorted[0];
        t.cmax = t.sorted[NC - 1];
        t.need_clamp = !(t.sorted[0] <= -1.0f && t.sorted[NC - 1] >= 1.0f);
    }
    if constexpr (NC == 256) {
        // signed cell number of each threshold: cell + kCells8 for q >= 0, kCells8 - 1 - cell below (non-decreasing in j)
        for (int j = tid; j < NC - 1; j += blockDim.x) {
            const unsigned u = __float_as_uint(t.thr[j]);
            const int c = cell8_of(u & 0x7fffffffu);          // may exceed kCells8 - 1: a threshold no quotient reaches
            t.thr_cell[j] = (u >> 31) ? kCells8 - 1 - c : kCells8 + c;
        }
        __syncthreads();
        for (int k = tid; k < 2 * kCells8; k += blockDim.x) {
            const bool neg = k < kCells8;                     // k in the order of q
            int lo = 0, hi = NC - 1;                          // first threshold whose cell is >= k
            while (lo < hi) { const int m = (lo + hi) >> 1; if (t.thr_cell[m] < k) lo = m + 1; else hi = m; }
            const int inside = (lo < NC - 1 && t.thr_cell[lo] == k) ? ((lo + 1 < NC - 1 && t.thr_cell[lo + 1] == k) ? 2 : 1) : 0;
            unsigned from = neg ? 0u : (1u << kCellShift8);   // no threshold in this cell
            if (inside) from = (__float_as_uint(t.thr[lo]) & ((1u << kCellShift8) - 1u)) + (neg ? 1u : 0u);
            const int cell = neg ? kCells8 - 1 - k : k - kCells8;
            // the lowest cell spans many binades: a threshold there is left to the search
            const unsigned slow = (inside > 1 || (inside == 1 && cell == 0)) ? 256u : 0u;
            t.lut8[(neg ? kCells8 : 0) + cell] = (from << 14) | slow | (unsigned)min(lo, 255);
        }
    }
    __syncthreads();
    if constexpr (NC == 16) {
        if (tid < NC - 1) t.thr_cell[tid] = __float_as_int(3.0f + t.thr[tid]);
        // the coarsest grid whose cells see at most one threshold each: few cells mean few distinct shared-memory words
        for (int cb = 7; cb <= kLutMaxBits; cb += 2) {
            if (tid == 0) { t.lut_bad = 0; t.lut_shift = 21 - cb; t.lut_mask = ((2u << cb) - 1u) << 2; }
            __syncthreads();
            bool bad = false;
            for (int k = tid; k <= (1 << cb); k += blockDim.x) {
                // a cell sees the thresholds inside it and up to four units of the last place beyond its borders
                const int lo = 0x40000000 + (k << (23 - cb)) - 4, hi = 0x40000000 + ((k + 1) << (23 - cb)) + 3;
                int base = 0, seen = 0, at = 0;
#pragma unroll
                for (int j = 0; j < NC - 1; ++j) {
                    const int c = t.thr_cell[j];
                    base += c < lo;
                    if (c >= lo && c <= hi) { ++seen; at = c; }
                }
                bad = bad || seen > 1;
                t.lut[k] = seen ? ((unsigned)(base + 1) << 24) + 4u - (unsigned)at
                                : ((unsigned)base << 24) + (1u << 22) - 0x40000000u;
            }
            if (!__syncthreads_or(bad)) break;
            if (tid == 0) t.lut_bad = 1;
        }
        __syncthreads();
    }
}

// Code of x / d in a sorted 16-entry codebook from one fused multiply-add: u = x * rcp + 3 with rcp = 1 / d rounded
// towards zero (|x| <= d, so u stays in [2, 4]) is within two units of its last place of 3 + x / d.  The top
// byte of the result is the code unless the lower 24 bits are at most 8, i.e. u is within four units of the cell's
// threshold: then (once in some 10^5 elements) the caller has to divide and search.
__device__ __forceinline__ unsigned code_word(const CodeTables<16> &t, int shift, unsigned mask, float x, float rcp) {
    const unsigned u = __float_as_uint(fmaf(x, rcp, 3.0f));
    return u + *reinterpret_cast<const unsigned *>(reinterpret_cast<const char *>(t.lut) + ((u >> shift) & mask));
}
// Eight codes in the top bytes of s -> one output word, element 2j in the high nibble of byte j (functional.py:733-734).
__device__ __forceinline__ unsigned pack_codes(const unsigned *s) {
    const unsigned e = __byte_perm(__byte_perm(s[0], s[2], 0x0073), __byte_perm(s[4], s[6], 0x0073), 0x5410);
    const unsigned o = __byte_perm(__byte_perm(s[1], s[3], 0x0073), __byte_perm(s[5], s[7], 0x0073), 0x5410);
    return (e << 4) | o;
}

// Number of thresholds <= q (== index into the sorted codebook).
template <int NC>
__device__ __forceinline__ int code_index_search(const CodeTables<NC> &t, float q) {
    int lo = 0;
#pragma unroll
    for (int step = NC / 2; step > 0; step >>= 1)
        if (t.thr[lo + step - 1] <= q) lo += step;
    return lo;
}

// x / d rounded to nearest, given r = RN(1/d): one reciprocal multiply and two FMA
// corrections (Markstein).  Exact whenever no intermediate underflows; callers guarantee
// 2^-40 <= d <= 2^60 and treat |quotient| < 2^-60 as "sign only" (see k_quantize_vec).
__device__ __forceinline__ float div_by_recip(float x, float d, float r) {
    float q = x * r;
    q = fmaf(fmaf(-q, d, x), r, q);
    q = fmaf(fmaf(-q, d, x), r, q);
    return q;
}

// Index of q = x / d (exact, |q| <= 1) in a 256-entry codebook; `slow` collects the cells that need the search.
__device__ __forceinline__ unsigned lut8_index(const unsigned *lut, float q, unsigned &slow) {
    const unsigned u = __float_as_uint(q), mag = u & 0x7fffffffu, neg = u >> 31;
    const unsigned e = lut[(neg ? kCells8 : 0) + cell8_of(mag)];
    slow |= e & 256u;
    return (e & 255u) + (((mag & ((1u << kCellShift8) - 1u)) >= (e >> 14) ? 1u : 0u) ^ neg);
}

// Exponent of a scaled fp16 operand plane: with amax = m * 2^k, m in [0.5, 1), e = target - k puts
// the largest scaled entry just below 2^target (0 for an all-zero or non-finite matrix).
__device__ __forceinline__ int exponent_for(float amax, int target) {
    if (!(amax > 0.0f) || !(amax <= 3.0e38f)) return 0;
    int k;
    frexpf(amax, &k);
    return target - k;
}

// Per-lane quantization of EPL elements for every case the lean path of k_quantize_vec does
// not cover (any codebook, clamp, permutation, extreme scales).  Kept out of line on purpose.
// Operands and results travel by value (registers): passing the caller's arrays by reference
// would force them into local memory on the hot path as well.
template <int EPL> struct LaneVals { float v[EPL]; };

template <int NC, int EPL>
__device__ __noinline__ unsigned long long quantize_lane_generic(const CodeTables<NC> &tab, LaneVals<EPL> x, float amax) {
    unsigned long long packed = 0;                        // one byte per element
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        int k = 0;
        if (amax != 0.0f) {
            float q = __fdiv_rn(x.v[j], amax);
            if (tab.need_clamp) q = fminf(fmaxf(q, tab.cmin), tab.cmax);
            const int idx = code_index_search<NC>(tab, q);
            k = tab.perm[idx];
        }
        packed |= (unsigned long long)(unsigned)k << (8 * j);
    }
    return packed;
}

}  // namespace qt
