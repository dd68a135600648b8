// Blockwise low-bit quantize / dequantize of square matrices for sm_100a.
//
// Semantics follow the reference's CPU quantizer (reference project paths):
//   qtensor/functional.py:526-615 (_quantize_blockwise_cpu), :618-688
//   (_dequantize_blockwise_cpu), :703-715 (_nearest_code_indices), :718-746 (nibble
//   packing) - and replace the CUDA kernels of cudaC_python/csrc/kernels.cu:57-457.
//
// Design (HBM-bound byte work, no tensor cores):
//   * one launch covers a strided batch of same-order matrices (quantize: one resident wave
//     of CTAs striding over the blocks of the whole batch; dequantize: gridDim.y = matrix);
//   * a quantization block (64..256 elements of one row) is owned by a group of LPU
//     lanes of one warp, EPL consecutive elements per lane, loaded as 128-bit vectors;
//     the per-block absmax is a shuffle reduction inside the group;
//   * the nearest-code rule |q-c_lo| > |c_hi-q| (fp32) is monotone in q, so it is
//     replaced by 2^bits-1 exact fp32 thresholds found once per CTA by bisection over
//     float bit patterns; the code index is the number of thresholds <= q.  A lookup table in
//     shared memory over cells of q resolves an element with one LDS.32 and one add or compare;
//   * q = x / absmax is an IEEE-rounded fp32 division (the oracle divides);
//   * codes are packed high-nibble-first and stored as 32/64-bit words.
//   Orders that are not a multiple of 8, unaligned buffers and block sizes above 256 take kernels that
//   work on the flat element stream, eight elements per thread whatever rows they belong to
//   (k_quantize_rows, k_dequantize_flat).
#include "quant_device.cuh"
#include <cuda_fp16.h>

namespace qt {

static constexpr int kThreads = 256;

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// 256-bit global accesses (sm_100): one request per lane for 32 bytes, half the L1 wavefronts of
// two 128-bit ones.  The address must be 32-byte aligned.
__device__ __forceinline__ void ldg256(const void *p, unsigned (&w)[8]) {
    asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "l"(p));
}
__device__ __forceinline__ void stg256(void *p, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 :: "l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
// 8 consecutive elements from a 32-byte (fp32) or 16-byte (bf16) aligned address.
template <typename T>
__device__ __forceinline__ void load8_wide(const T *p, float *x) {
    if constexpr (sizeof(T) == 4) {
        unsigned w[8];
        ldg256(p, w);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(w[j]);
    } else {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p));
        const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            x[2 * j] = __uint_as_float(w[j] << 16);
            x[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
        }
    }
}

// Load EPL (8 or 16) consecutive elements from a 16-byte aligned address.
template <typename T, int EPL>
__device__ __forceinline__ void load_vec(const T *p, float (&x)[EPL]) {
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int j = 0; j < EPL; j += 4) {
            float4 v = __ldg(reinterpret_cast<const float4 *>(p + j));
            x[j] = v.x; x[j + 1] = v.y; x[j + 2] = v.z; x[j + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int h = 0; h < EPL / 8; ++h) {
            uint4 v = __ldg(reinterpret_cast<const uint4 *>(p + 8 * h));
            unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                x[8 * h + 2 * j] = __uint_as_float(w[j] << 16);
                x[8 * h + 2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
            }
        }
    }
}

// ------------------------------------------------------------------------------------
// Quantize, vector path.  Requires n % EPL == 0 and vector-aligned buffers.
// ------------------------------------------------------------------------------------
template <typename T, int BITS, int EPL, int LPU>
__global__ void __launch_bounds__(kThreads, 4)
k_quantize_vec(const T *__restrict__ Abase, long long strideA, const float *__restrict__ code,
               int n, int nb, int count, float *__restrict__ absmax_base, long long stride_absmax,
               float *__restrict__ diag_base, long long stride_diag,
               unsigned char *__restrict__ out_base, long long stride_out, int wide) {
    constexpr int NC = 1 << BITS;
    constexpr int BS = EPL * LPU;
    // EPL == 16: a lane holds two octets of its block, 8 LPU columns apart, so that one load instruction of the
    // LPU lanes covers whole 128-byte lines (with 16 consecutive elements per lane the same lines were looked up by two
    // instructions and L1 was the bound: 125 x 768^2 83 -> 74 us, 0.71 of the measured copy rate).
    // `wide`: octets of fp32 start on a 32-byte boundary.
    constexpr int STEP = 8 * LPU;
    auto load_lane = [&](const T *p, int c, float (&dst)[EPL]) {
        if constexpr (EPL == 16) {
            if (wide) {
                load8_wide<T>(p, dst);
                if (c + STEP < n) load8_wide<T>(p + STEP, dst + 8);
                else {
#pragma unroll
                    for (int j = 8; j < 16; ++j) dst[j] = 0.0f;
                }
                return;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float y[8];
                if (c + h * STEP < n) load_vec<T, 8>(p + h * STEP, y);
#pragma unroll
                for (int j = 0; j < 8; ++j) dst[8 * h + j] = c + h * STEP < n ? y[j] : 0.0f;
            }
        } else {
            load_vec<T, EPL>(p, dst);
        }
    };
    __shared__ CodeTables<NC> tab;

    // A warp works on one block column of GW consecutive rows (a "warp unit": GW quantization
    // blocks, LPU lanes each), so the diagonal crosses only one warp unit in nb and the diagonal
    // side channel costs nothing elsewhere.  Warp units are numbered across the whole batch
    // (matrix, row band, block); the grid is one resident wave (the tables are built once per CTA and no
    // second wave trails behind) and every warp takes a run of consecutive units, so that stepping to the
    // next one is three additions except at the end of a band.
    constexpr int GW = 32 / LPU;
    const int bands = (n + GW - 1) / GW;
    const int wunits = bands * nb;                          // per matrix
    const int total = wunits * count;                       // launcher keeps this below 2^31
    const int W = gridDim.x * (kThreads / 32), wid = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int lane_u = threadIdx.x % LPU, row_in_band = (threadIdx.x & 31) / LPU;
    const int share = total / W, extra = total - share * W;
    int left = share + (wid < extra ? 1 : 0);                // units of this warp
    const int first = wid * share + min(wid, extra);
    int m = first / wunits;
    int band = (first - m * wunits) / nb, b = first - m * wunits - band * nb;
    int r, c;
    long long eo, ao;                                        // element offset of this lane, scale offset of its block (within the matrix)
    auto place = [&]() {
        r = band * GW + row_in_band;
        c = b * BS + lane_u * 8;
        eo = (long long)r * n + c;
        ao = (long long)r * nb + b;
    };
    place();

    // the first loads are issued before the table build so that its latency is hidden
    float xn[EPL];
    auto fetch = [&]() {
        if (left > 0 && r < n && c < n) { load_lane(Abase + (long long)m * strideA + eo, c, xn); return; }
#pragma unroll
        for (int j = 0; j < EPL; ++j) xn[j] = 0.0f;
    };
    fetch();
    build_tables<NC>(tab, code);
    const bool lean_launch = !tab.lut_bad && !tab.need_clamp && tab.perm_identity && !tab.tiny_thr;
    const int lut_shift = tab.lut_shift;
    const unsigned lut_mask = tab.lut_mask;

    while (left > 0) {
        const int cr = r, cc = c;
        const long long cm = m, e = eo, ca = ao;              // e: flat element index, multiple of 8
        const bool unit_ok = cr < n;
        const bool lane_ok = unit_ok && cc < n;
        float x[EPL];
#pragma unroll
        for (int j = 0; j < EPL; ++j) x[j] = xn[j];
        // the loads of this warp's next unit are in flight while this one is encoded
        --left;
        if (++b < nb) { c += BS; eo += BS; ao += 1; }
        else {
            b = 0;
            if (++band == bands) { band = 0; ++m; }
            place();
        }
        fetch();
        if (diag_base && lane_ok && (unsigned)(cr - cc) < (unsigned)BS) {   // functional.py:574-578
#pragma unroll
            for (int j = 0; j < EPL; ++j)
                if (cc + (j & 7) + (j >> 3) * STEP == cr) { diag_base[cm * stride_diag + cr] = x[j]; x[j] = 0.0f; }
        }
        float amax = 0.0f;
#pragma unroll
        for (int j = 0; j < EPL; ++j) amax = fmaxf(amax, fabsf(x[j]));
#pragma unroll
        for (int off = LPU / 2; off > 0; off >>= 1)
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        if (unit_ok && lane_u == 0) absmax_base[cm * stride_absmax + ca] = amax;

        // Lean path (the hot one: sorted codebook covering [-1, 1], no threshold within 2^-50 of zero, block
        // scale in [2^-40, 2^60] or zero).  4 bits: code_word(); 8 bits: the exact quotient from a
        // reciprocal and two FMA corrections - bit-identical to the IEEE division (functional.py:604) while nothing
        // underflows; a |q| below 2^-60 only has to keep its sign.  Anything else takes the out-of-line routine.
        const bool lean = lean_launch && ((amax >= 9.094947e-13f && amax <= 1.1529215e18f) || amax == 0.0f);
        if (lane_ok) {
            unsigned char *out = out_base + cm * stride_out;
            if constexpr (BITS == 4) {
                constexpr int NW = EPL / 8;
                unsigned wq[NW];
#pragma unroll
                for (int i = 0; i < NW; ++i) wq[i] = 0;
                bool generic = !lean;
                if (lean && amax != 0.0f) {                    // an all-zero block has codes 0 (functional.py:600-602)
                    const float rcp = __frcp_rz(amax);
                    unsigned nearest = 0xffffffffu;
#pragma unroll
                    for (int i = 0; i < NW; ++i) {
                        unsigned w[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            w[j] = code_word(tab, lut_shift, lut_mask, x[8 * i + j], rcp);
                            nearest = min(nearest, w[j] & 0xffffffu);
                        }
                        wq[i] = pack_codes(w);
                    }
                    generic = nearest <= 8u;                  // rare: redo this lane with the exact division
                }
                if (generic) {
#pragma unroll
                    for (int h = 0; h < NW; ++h) {
                        LaneVals<8> xv;
#pragma unroll
                        for (int j = 0; j < 8; ++j) xv.v[j] = x[h * 8 + j];
                        const unsigned long long pk = quantize_lane_generic<NC, 8>(tab, xv, amax);
                        unsigned w[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) w[j] = (unsigned)(pk >> (8 * j)) << 24;
                        wq[h] = pack_codes(w);
                    }
                }
                *reinterpret_cast<unsigned *>(out + (e >> 1)) = wq[0];
                if constexpr (EPL == 16)
                    if (cc + STEP < n) *reinterpret_cast<unsigned *>(out + (e >> 1) + STEP / 2) = wq[1];
            } else {
                unsigned w0 = 0, w1 = 0;
                bool generic = !lean;
                if (lean && amax != 0.0f) {
                    const float rcp = __frcp_rn(amax);
                    unsigned slow = 0;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        w0 |= lut8_index(tab.lut8, div_by_recip(x[j], amax, rcp), slow) << (8 * j);
                        w1 |= lut8_index(tab.lut8, div_by_recip(x[4 + j], amax, rcp), slow) << (8 * j);
                    }
                    generic = slow != 0u;
                }
                if (generic) {
                    LaneVals<8> xv;
#pragma unroll
                    for (int j = 0; j < 8; ++j) xv.v[j] = x[j];
                    const unsigned long long pk = quantize_lane_generic<NC, 8>(tab, xv, amax);
                    w0 = (unsigned)pk; w1 = (unsigned)(pk >> 32);
                }
                *reinterpret_cast<uint2 *>(out + e) = make_uint2(w0, w1);
            }
        }
    }
}

// ------------------------------------------------------------------------------------
// Quantize, any order, alignment and block size.  A CTA takes eight rows at a time: eight rows start and end on a
// multiple of eight elements of the flat stream, so that however odd the order is, whole output words belong to
// one CTA.  First the scales of the rows' blocks (one warp per row, 256 columns in flight), kept in shared memory with
// their reciprocals; then the codes, eight consecutive elements of the stream per thread (the second read of
// the rows comes from L1 / L2).  Such an octet lies in one or two quantization blocks; in three where a row ends in a
// block shorter than the octet (left to the search).  The grid is one resident wave: each CTA builds the code tables once.
// Bound by instruction issue (58 % of the slots) and, for a single small matrix, by the chain build - scales - codes of
// its 2.5 CTAs per SM.  Measured against a pass for the scales and one thread per output byte: 3001^2 bf16, 8 bits, block
// 256: 224 -> 43 us; 8 x 1189^2, 4 bits: 99 -> 41; 8191^2, 4 bits: 462 -> 142.
// ------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void load8(const T *p, int nvalid, bool vec, float (&x)[8]) {
    if (vec && nvalid == 8) { load_vec<T, 8>(p, x); return; }
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = j < nvalid ? to_f32<T>(p[j]) : 0.0f;
}

// Eight consecutive elements of the flat stream of an n x n matrix (n >= 8), row r and column c of the first; elements
// [0, first) lie in its quantization block, [first, second) in the next one, the rest in the one after.
struct Octet { int r, c, first, second; };
__device__ __forceinline__ Octet octet_at(int r, int c, int n, int bs_shift) {
    Octet o;
    o.r = r;
    o.c = c;
    const int row_left = n - o.c;
    o.first = min(8, min(row_left, (((o.c >> bs_shift) + 1) << bs_shift) - o.c));
    o.second = o.first < row_left ? min(8, row_left) : 8;     // a row's first block has at least eight elements
    return o;
}
// Position of the diagonal element inside the octet (8 or more: none).
__device__ __forceinline__ int octet_diag(const Octet &o, int n) {
    const int here = o.r - o.c, next = n - o.c;              // `next`: position of the following row's first element
    if (here >= 0 && here < min(8, next)) return here;
    return next < 8 ? next + o.r + 1 : 8;                     // column r + 1 of row r + 1
}

template <typename T, int BITS>
__global__ void __launch_bounds__(kThreads, 4)
k_quantize_rows(const T *__restrict__ Abase, long long strideA, const float *__restrict__ code,
                int n, int nb, int bs_shift, int groups, int count, float *__restrict__ absmax_base, long long stride_absmax,
                float *__restrict__ diag_base, long long stride_diag, unsigned char *__restrict__ out_base, long long stride_out,
                int vec_in, int vec_out) {
    constexpr int NC = 1 << BITS;
    __shared__ CodeTables<NC> tab;
    extern __shared__ float2 scale_s[];                      // [8 * nb]: block scales of the eight rows and their reciprocals
    build_tables<NC>(tab, code);
    const bool lean_launch = !tab.lut_bad && !tab.need_clamp && tab.perm_identity && !tab.tiny_thr;
    const int lut_shift = tab.lut_shift;
    const unsigned lut_mask = tab.lut_mask;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int dr = (8 * kThreads) / n, dc = 8 * kThreads - dr * n;
    for (int work = blockIdx.x; work < groups * count; work += gridDim.x) {
        const int m = work / groups, r0 = (work - m * groups) * 8, rows = min(8, n - r0);
        const T *A = Abase + (long long)m * strideA;
        unsigned char *out = out_base + (long long)m * stride_out;
        if (warp < rows) {
            const int r = r0 + warp;
            const T *row = A + (long long)r * n;
            float *absmax = absmax_base + (long long)m * stride_absmax + (long long)r * nb;
            const int per = bs_shift >= 8 ? 1 : 256 >> bs_shift;           // blocks in 256 columns
            float wide_max = 0.0f;                            // blocks above 256: maximum so far
            T xn[8];                                          // the next 256 columns are in flight while these are reduced
            auto fetch = [&](int c0) {
#pragma unroll
                for (int k = 0; k < 8; ++k) xn[k] = c0 + 32 * k + lane < n ? row[c0 + 32 * k + lane] : T(0.0f);
            };
            fetch(0);
            for (int c0 = 0; c0 < n; c0 += 256) {
                float x[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) x[k] = to_f32<T>(xn[k]);
                fetch(c0 + 256);
                if (diag_base && (unsigned)(r - c0) < 256u) {
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (c0 + 32 * k + lane == r) { diag_base[(long long)m * stride_diag + r] = x[k]; x[k] = 0.0f; }
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) x[k] = fabsf(x[k]);
#pragma unroll
                for (int k = 0; k < 4; ++k) x[k] = fmaxf(x[2 * k], x[2 * k + 1]);
                if (per <= 2) { x[0] = fmaxf(x[0], x[1]); x[1] = fmaxf(x[2], x[3]); }
                if (per == 1) x[0] = fmaxf(x[0], x[1]);
                // magnitudes order like their bit patterns: warp-wide integer maxima
                float amax = 0.0f;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k < per) {
                        const float v = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(x[k])));
                        if (lane == k) amax = v;
                    }
                if (bs_shift > 8) {
                    wide_max = fmaxf(wide_max, amax);
                    if (((c0 + 256) & ((1 << bs_shift) - 1)) && c0 + 256 < n) continue;
                    amax = wide_max;
                    wide_max = 0.0f;
                }
                const int b = (c0 >> bs_shift) + lane;
                if (lane < per && b < nb) {
                    // reciprocal 0: not for the lean path (an all-zero block, or a scale outside [2^-40, 2^60])
                    const bool plain = lean_launch && amax >= 9.094947e-13f && amax <= 1.1529215e18f;
                    scale_s[warp * nb + b] = make_float2(amax, plain ? (BITS == 4 ? __frcp_rz(amax) : __frcp_rn(amax)) : 0.0f);
                    absmax[b] = amax;
                }
            }
        }
        __syncthreads();
        const unsigned e_begin = (unsigned)r0 * (unsigned)n, e_end = e_begin + (unsigned)rows * (unsigned)n;   // below 2^31
        int rr = (8 * threadIdx.x) / n, cc = 8 * threadIdx.x - rr * n;      // row within the group and column of the octet
        float xn[8];
        unsigned e = e_begin + 8u * threadIdx.x;
        if (e < e_end) load8<T>(A + e, (int)min(8u, e_end - e), vec_in != 0, xn);
        for (; e < e_end; e += 8u * kThreads) {
            const int nvalid = (int)min(8u, e_end - e);
            const Octet o = octet_at(r0 + rr, cc, n, bs_shift);
            float x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = xn[j];
            const unsigned e2 = e + 8u * kThreads;
            if (e2 < e_end) load8<T>(A + e2, (int)min(8u, e_end - e2), vec_in != 0, xn);
            const int u0 = rr * nb + (cc >> bs_shift);
            const float2 s0 = scale_s[u0], s1 = o.first < nvalid ? scale_s[u0 + 1] : s0;
            if (diag_base) {
                const int jd = octet_diag(o, n);
#pragma unroll
                for (int j = 0; j < 8; ++j) if (j == jd) x[j] = 0.0f;
            }
            unsigned idx[8];                                   // codes (4 bits: in the top byte)
            unsigned slow = (s0.y != 0.0f && s1.y != 0.0f && o.second >= nvalid) ? 0u : 1u;
            if (!slow) {
                unsigned nearest = 0xffffffffu;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const bool in0 = j < o.first;
                    if constexpr (BITS == 4) {
                        idx[j] = code_word(tab, lut_shift, lut_mask, x[j], in0 ? s0.y : s1.y);
                        nearest = min(nearest, idx[j] & 0xffffffu);
                    } else {
                        idx[j] = lut8_index(tab.lut8, div_by_recip(x[j], in0 ? s0.x : s1.x, in0 ? s0.y : s1.y), slow);
                    }
                }
                if (BITS == 4 && nearest <= 8u) slow = 1u;
            }
            if (slow) {
                LaneVals<8> xv;
#pragma unroll
                for (int j = 0; j < 8; ++j) xv.v[j] = x[j];
                const unsigned long long p0 = quantize_lane_generic<NC, 8>(tab, xv, s0.x);
                const unsigned long long p1 = o.first < nvalid ? quantize_lane_generic<NC, 8>(tab, xv, s1.x) : p0;
                const unsigned long long p2 = o.second < nvalid ? quantize_lane_generic<NC, 8>(tab, xv, scale_s[u0 + 2].x) : p0;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    idx[j] = ((unsigned)((j < o.first ? p0 : j < o.second ? p1 : p2) >> (8 * j)) & 255u) << (BITS == 4 ? 24 : 0);
            }
            if (nvalid < 8) {
#pragma unroll
                for (int j = 0; j < 8; ++j) if (j >= nvalid) idx[j] = 0;  // a padding nibble is 0 (functional.py:724-732)
            }
            rr += dr; cc += dc;
            if (cc >= n) { cc -= n; ++rr; }
            if constexpr (BITS == 4) {
                const unsigned w = pack_codes(idx);
                unsigned char *dst = out + (e >> 1);
                if (vec_out && nvalid == 8) *reinterpret_cast<unsigned *>(dst) = w;
                else for (int j = 0; j < (nvalid + 1) / 2; ++j) dst[j] = (unsigned char)(w >> (8 * j));
            } else {
                unsigned w0 = 0, w1 = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) { w0 |= idx[j] << (8 * j); w1 |= idx[4 + j] << (8 * j); }
                unsigned char *dst = out + e;
                if (vec_out && nvalid == 8) *reinterpret_cast<uint2 *>(dst) = make_uint2(w0, w1);
                else for (int j = 0; j < nvalid; ++j) dst[j] = (unsigned char)(j < 4 ? w0 >> (8 * j) : w1 >> (8 * (j - 4)));
            }
        }
        __syncthreads();                                      // the scales are replaced next
    }
}

// Orders below 8, where eight elements may touch more than two rows: one thread per output byte, one CTA per matrix.
template <typename T, int BITS>
__global__ void __launch_bounds__(64)
k_quantize_tiny(const T *__restrict__ Abase, long long strideA, const float *__restrict__ code, int n,
                float *__restrict__ absmax_base, long long stride_absmax, float *__restrict__ diag_base, long long stride_diag,
                unsigned char *__restrict__ out_base, long long stride_out) {
    constexpr int NC = 1 << BITS, PER = 8 / BITS;
    __shared__ CodeTables<NC> tab;
    __shared__ float scale_s[8];
    build_tables<NC>(tab, code);
    const T *A = Abase + (long long)blockIdx.x * strideA;
    if (threadIdx.x < n) {                                    // one block per row
        const int r = threadIdx.x;
        float amax = 0.0f;
        for (int c = 0; c < n; ++c) {
            const float x = to_f32<T>(A[r * n + c]);
            if (diag_base && c == r) diag_base[(long long)blockIdx.x * stride_diag + r] = x;
            else amax = fmaxf(amax, fabsf(x));
        }
        scale_s[r] = amax;
        absmax_base[(long long)blockIdx.x * stride_absmax + r] = amax;
    }
    __syncthreads();
    const int byte = threadIdx.x, total = n * n;
    if (byte >= (total + PER - 1) / PER) return;
    unsigned v = 0;
    for (int h = 0; h < PER; ++h) {
        const int e = byte * PER + h;
        unsigned k = 0;
        if (e < total) {
            LaneVals<1> xv;
            xv.v[0] = (diag_base && e / n == e % n) ? 0.0f : to_f32<T>(A[e]);
            k = (unsigned)quantize_lane_generic<NC, 1>(tab, xv, scale_s[e / n]);
        }
        v = BITS == 4 ? ((v << 4) | k) : k;
    }
    out_base[(long long)blockIdx.x * stride_out + byte] = (unsigned char)v;
}

// ------------------------------------------------------------------------------------
// Dequantize.
// ------------------------------------------------------------------------------------
template <typename T, int EPL> __device__ __forceinline__ void store_vec(T *p, const float (&v)[EPL]);
template <> __device__ __forceinline__ void store_vec<float, 8>(float *p, const float (&v)[8]) {
    stg256(p, v);                                             // launcher guarantees 32-byte alignment
}
__device__ __forceinline__ unsigned pack_bf16x2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);           // .x = a (low half), .y = b
    return *reinterpret_cast<unsigned *>(&h);
}
template <> __device__ __forceinline__ void store_vec<__nv_bfloat16, 8>(__nv_bfloat16 *p, const float (&v)[8]) {
    *reinterpret_cast<uint4 *>(p) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]),
                                               pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}

// Vector path: n % EPL == 0, aligned buffers; any supported block size (power of two).
template <typename T, int BITS, int EPL>
__global__ void __launch_bounds__(kThreads)
k_dequantize_vec(const unsigned char *__restrict__ in_base, long long stride_in, const float *__restrict__ code,
                 int n, int nb, int bs_shift, const float *__restrict__ absmax_base, long long stride_absmax,
                 const float *__restrict__ diag_base, long long stride_diag,
                 T *__restrict__ out_base, long long stride_out) {
    constexpr int NC = 1 << BITS;
    __shared__ float2 pair_lut[BITS == 4 ? 256 : 1];          // byte -> (high-nibble value, low-nibble value)
    __shared__ float code_s[BITS == 8 ? 256 : 16];
    for (int i = threadIdx.x; i < NC; i += blockDim.x) code_s[i] = code[i];
    __syncthreads();
    if (BITS == 4)
        for (int i = threadIdx.x; i < 256; i += blockDim.x) pair_lut[i] = make_float2(code_s[i >> 4], code_s[i & 15]);
    __syncthreads();

    const int m = blockIdx.y;
    const unsigned char *in = in_base + (long long)m * stride_in;
    const float *absmax = absmax_base + (long long)m * stride_absmax;
    const float *diag = diag_base ? diag_base + (long long)m * stride_diag : nullptr;
    T *out = out_base + (long long)m * stride_out;

    const int chunks_per_row = n / EPL;
    const int chunks = n * chunks_per_row;
    const int S = gridDim.x * kThreads;
    int t = blockIdx.x * kThreads + threadIdx.x;
    int r = t / chunks_per_row, cc = t - r * chunks_per_row;
    const int dr = S / chunks_per_row, dc = S - dr * chunks_per_row;
#pragma unroll 4
    for (; t < chunks; t += S) {
        const int c = cc * EPL;
        const long long e = (long long)r * n + c;
        const float amax = __ldg(absmax + (long long)r * nb + (c >> bs_shift));
        const float z = (amax == 0.0f) ? 0.0f : -0.0f;        // exact +0.0 for all-zero blocks (functional.py:663-665)
        float v[EPL];
        if constexpr (BITS == 4) {
            unsigned w;
            if constexpr (EPL == 8) w = __ldg(reinterpret_cast<const unsigned *>(in + (e >> 1)));
            else w = __ldg(reinterpret_cast<const unsigned short *>(in + (e >> 1)));
#pragma unroll
            for (int j = 0; j < EPL / 2; ++j) {
                float2 p = pair_lut[(w >> (8 * j)) & 255u];
                v[2 * j] = fmaf(p.x, amax, z);
                v[2 * j + 1] = fmaf(p.y, amax, z);
            }
        } else {
            unsigned w0, w1 = 0;
            if constexpr (EPL == 8) {
                uint2 ww = __ldg(reinterpret_cast<const uint2 *>(in + e));
                w0 = ww.x; w1 = ww.y;
            } else {
                w0 = __ldg(reinterpret_cast<const unsigned *>(in + e));
            }
#pragma unroll
            for (int j = 0; j < EPL; ++j) {
                unsigned byte = ((j < 4 ? w0 : w1) >> (8 * (j & 3))) & 255u;
                v[j] = fmaf(code_s[byte], amax, z);
            }
        }
        if (diag && r >= c && r < c + EPL) {                  // functional.py:673-678
            const float d = diag[r];
#pragma unroll
            for (int j = 0; j < EPL; ++j)
                if (c + j == r) v[j] = d;
        }
        store_vec<T, EPL>(out + e, v);
        r += dr; cc += dc;
        if (cc >= chunks_per_row) { cc -= chunks_per_row; r += 1; }
    }
}

// ------------------------------------------------------------------------------------
// Dequantize straight into the operand format of the tcgen05 products: two bf16 planes
// (hi = bf16(x), lo = bf16(x - hi)) with row pitch ldp.  Output matrix j is taken from state
// slot slots[j] (or j when slots == nullptr), so a product's batch can be assembled from
// scattered slots of an arena without an fp32 copy, a stack and a split pass in between.
// EPL = 8 elements per thread (one 32/64-bit code load, one 128-bit store per plane) or, with
// 32-byte aligned rows, 16 (one 256-bit store per plane).
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void stg256u(void *p, const unsigned (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 :: "l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

// Largest magnitude a dequantized state matrix can hold: max over its block scales and its fp32
// diagonal (|code| <= 1).  One CTA per output matrix; amax[m] belongs to state slot slots[m].
__global__ void __launch_bounds__(256)
k_state_amax(const float *__restrict__ absmax_base, long long stride_absmax, int n_absmax,
             const float *__restrict__ diag_base, long long stride_diag, int n_diag,
             const int *__restrict__ slots, float *__restrict__ amax, int *__restrict__ exp_out = nullptr, int target = 0) {
    const int m = blockIdx.x;
    const long long src = slots ? (long long)slots[m] : (long long)m;
    // four independent loads in flight per thread: a matrix has 9 K - 23 K block scales and this CTA is
    // alone with them, so the loop is bound by load latency, not bandwidth
    float v0 = 0.0f, v1 = 0.0f, v2 = 0.0f, v3 = 0.0f;
    const float *am = absmax_base + src * stride_absmax;
    const int step = blockDim.x;
    int i = threadIdx.x;
    for (; i + 3 * step < n_absmax; i += 4 * step) {
        const float a = __ldg(am + i), b = __ldg(am + i + step), c = __ldg(am + i + 2 * step), d = __ldg(am + i + 3 * step);
        v0 = fmaxf(v0, fabsf(a)); v1 = fmaxf(v1, fabsf(b)); v2 = fmaxf(v2, fabsf(c)); v3 = fmaxf(v3, fabsf(d));
    }
    for (; i < n_absmax; i += step) v0 = fmaxf(v0, fabsf(__ldg(am + i)));
    float v = fmaxf(fmaxf(v0, v1), fmaxf(v2, v3));
    if (diag_base)
        for (int k = threadIdx.x; k < n_diag; k += blockDim.x) v = fmaxf(v, fabsf(__ldg(diag_base + src * stride_diag + k)));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    __shared__ float red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i) v = fmaxf(v, red[i]);
        if (amax) amax[m] = v;
        if (exp_out) exp_out[m] = exponent_for(v, target);
    }
}

// F16: the planes are scaled fp16 planes (entry = value * 2^e, e from amax[m] and `target`,
// written to exp_out[m]); otherwise plain bf16 planes.
template <int BITS, int EPL, bool F16>
__global__ void __launch_bounds__(kThreads)
k_dequantize_planes(const unsigned char *__restrict__ in_base, long long stride_in, const float *__restrict__ code,
                    int n, int nb, int bs_shift, const float *__restrict__ absmax_base, long long stride_absmax,
                    const float *__restrict__ diag_base, long long stride_diag, const int *__restrict__ slots,
                    __nv_bfloat16 *__restrict__ hi_base, __nv_bfloat16 *__restrict__ lo_base, long long ldp, long long strideP,
                    const float *__restrict__ amax, int target, int *__restrict__ exp_out) {
    constexpr int NC = 1 << BITS;
    __shared__ float2 pair_lut[BITS == 4 ? 256 : 1];
    __shared__ float code_s[BITS == 8 ? 256 : 16];
    for (int i = threadIdx.x; i < NC; i += blockDim.x) code_s[i] = code[i];
    __syncthreads();
    if (BITS == 4)
        for (int i = threadIdx.x; i < 256; i += blockDim.x) pair_lut[i] = make_float2(code_s[i >> 4], code_s[i & 15]);
    __syncthreads();

    const int m = blockIdx.y;
    const long long src = slots ? (long long)slots[m] : (long long)m;
    const unsigned char *in = in_base + src * stride_in;
    const float *absmax = absmax_base + src * stride_absmax;
    const float *diag = diag_base ? diag_base + src * stride_diag : nullptr;
    __nv_bfloat16 *hi = hi_base + (long long)m * strideP, *lo = lo_base + (long long)m * strideP;
    float two_e = 1.0f;
    if constexpr (F16) {
        const int e = exponent_for(amax[m], target);
        two_e = exp2f((float)e);
        if (exp_out && blockIdx.x == 0 && threadIdx.x == 0) exp_out[m] = e;
    }

    const int chunks_per_row = n / EPL;
    const int chunks = n * chunks_per_row;
    const int S = gridDim.x * kThreads;
    int t = blockIdx.x * kThreads + threadIdx.x;
    int r = t / chunks_per_row, cc = t - r * chunks_per_row;
    const int dr = S / chunks_per_row, dc = S - dr * chunks_per_row;
#pragma unroll 2
    for (; t < chunks; t += S) {
        const int c = cc * EPL;
        const long long e = (long long)r * n + c;
        const float amax = __ldg(absmax + (long long)r * nb + (c >> bs_shift));
        const float z = (amax == 0.0f) ? 0.0f : -0.0f;        // exact +0.0 for all-zero blocks
        float v[EPL];
        if constexpr (BITS == 4) {
            unsigned w[EPL / 8];
            if constexpr (EPL == 16) {
                const uint2 ww = __ldg(reinterpret_cast<const uint2 *>(in + (e >> 1)));
                w[0] = ww.x; w[1] = ww.y;
            } else {
                w[0] = __ldg(reinterpret_cast<const unsigned *>(in + (e >> 1)));
            }
#pragma unroll
            for (int j = 0; j < EPL / 2; ++j) {
                const float2 pr = pair_lut[(w[j / 4] >> (8 * (j & 3))) & 255u];
                v[2 * j] = fmaf(pr.x, amax, z);
                v[2 * j + 1] = fmaf(pr.y, amax, z);
            }
        } else {
            unsigned w[EPL / 4];
            if constexpr (EPL == 16) {
                const uint4 ww = __ldg(reinterpret_cast<const uint4 *>(in + e));
                w[0] = ww.x; w[1] = ww.y; w[2] = ww.z; w[3] = ww.w;
            } else {
                const uint2 ww = __ldg(reinterpret_cast<const uint2 *>(in + e));
                w[0] = ww.x; w[1] = ww.y;
            }
#pragma unroll
            for (int j = 0; j < EPL; ++j) v[j] = fmaf(code_s[(w[j / 4] >> (8 * (j & 3))) & 255u], amax, z);
        }
        if (diag && (unsigned)(r - c) < (unsigned)EPL) {
            const float d = diag[r];
#pragma unroll
            for (int j = 0; j < EPL; ++j)
                if (c + j == r) v[j] = d;
        }
        unsigned h[EPL / 2], l[EPL / 2];
#pragma unroll
        for (int j = 0; j < EPL / 2; ++j) {
            if constexpr (F16) {
                const float a0 = v[2 * j] * two_e, a1 = v[2 * j + 1] * two_e;
                const __half h0 = __float2half_rn(a0), h1 = __float2half_rn(a1);
                const __half l0 = __float2half_rn(a0 - __half2float(h0)), l1 = __float2half_rn(a1 - __half2float(h1));
                h[j] = (unsigned)__half_as_ushort(h0) | ((unsigned)__half_as_ushort(h1) << 16);
                l[j] = (unsigned)__half_as_ushort(l0) | ((unsigned)__half_as_ushort(l1) << 16);
            } else {
                const __nv_bfloat16 h0 = __float2bfloat16_rn(v[2 * j]), h1 = __float2bfloat16_rn(v[2 * j + 1]);
                const __nv_bfloat16 l0 = __float2bfloat16_rn(v[2 * j] - __bfloat162float(h0));
                const __nv_bfloat16 l1 = __float2bfloat16_rn(v[2 * j + 1] - __bfloat162float(h1));
                h[j] = (unsigned)__bfloat16_as_ushort(h0) | ((unsigned)__bfloat16_as_ushort(h1) << 16);
                l[j] = (unsigned)__bfloat16_as_ushort(l0) | ((unsigned)__bfloat16_as_ushort(l1) << 16);
            }
        }
        const long long o = (long long)r * ldp + c;
        if constexpr (EPL == 16) {
            stg256u(hi + o, h);
            stg256u(lo + o, l);
        } else {
            *reinterpret_cast<uint4 *>(hi + o) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4 *>(lo + o) = make_uint4(l[0], l[1], l[2], l[3]);
        }
        r += dr; cc += dc;
        if (cc >= chunks_per_row) { cc -= chunks_per_row; r += 1; }
    }
}

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Any order and alignment: eight consecutive elements of the flat stream per thread (see k_quantize_rows), one vector
// load and store each; 3001^2 bf16, 8 bits: 45 -> 18 us with one element per thread before.
template <typename T, int BITS>
__global__ void __launch_bounds__(kThreads)
k_dequantize_flat(const unsigned char *__restrict__ in_base, long long stride_in, const float *__restrict__ code,
                  int n, int nb, int bs_shift, const float *__restrict__ absmax_base, long long stride_absmax,
                  const float *__restrict__ diag_base, long long stride_diag,
                  T *__restrict__ out_base, long long stride_out, int vec_in, int vec_out) {
    constexpr int NC = 1 << BITS;
    __shared__ float code_s[NC];
    for (int i = threadIdx.x; i < NC; i += blockDim.x) code_s[i] = code[i];
    __syncthreads();
    const int m = blockIdx.y;
    const unsigned char *in = in_base + (long long)m * stride_in;
    const float *absmax = absmax_base + (long long)m * stride_absmax;
    const float *diag = diag_base ? diag_base + (long long)m * stride_diag : nullptr;
    T *out = out_base + (long long)m * stride_out;
    const unsigned total = (unsigned)n * (unsigned)n;         // below 2^31
#pragma unroll 2
    for (unsigned e = 8u * (blockIdx.x * kThreads + threadIdx.x); e < total; e += 8u * kThreads * gridDim.x) {
        const int nvalid = (int)min(8u, total - e);
        unsigned idx[8];
        if constexpr (BITS == 4) {
            const unsigned char *src = in + (e >> 1);
            unsigned w = 0;
            if (vec_in && nvalid == 8) w = __ldg(reinterpret_cast<const unsigned *>(src));
            else for (int j = 0; j < (nvalid + 1) / 2; ++j) w |= (unsigned)src[j] << (8 * j);
#pragma unroll
            for (int j = 0; j < 8; j += 2) { idx[j] = (w >> (4 * j + 4)) & 15u; idx[j + 1] = (w >> (4 * j)) & 15u; }
        } else {
            const unsigned char *src = in + e;
            uint2 w = make_uint2(0u, 0u);
            if (vec_in && nvalid == 8) w = __ldg(reinterpret_cast<const uint2 *>(src));
            else for (int j = 0; j < nvalid; ++j) { if (j < 4) w.x |= (unsigned)src[j] << (8 * j); else w.y |= (unsigned)src[j] << (8 * (j - 4)); }
#pragma unroll
            for (int j = 0; j < 4; ++j) { idx[j] = (w.x >> (8 * j)) & 255u; idx[4 + j] = (w.y >> (8 * j)) & 255u; }
        }
        float v[8];
        if (n >= 8) {
            const int r = (int)(e / (unsigned)n);
            const Octet o = octet_at(r, (int)(e - (unsigned)r * (unsigned)n), n, bs_shift);
            const long long u0 = (long long)o.r * nb + (o.c >> bs_shift);
            const float am0 = __ldg(absmax + u0), am1 = o.first < nvalid ? __ldg(absmax + u0 + 1) : am0;
            const float am2 = o.second < nvalid ? __ldg(absmax + u0 + 2) : am0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float am = j < o.first ? am0 : j < o.second ? am1 : am2;
                v[j] = fmaf(code_s[idx[j]], am, am == 0.0f ? 0.0f : -0.0f);   // exact +0.0 for all-zero blocks (functional.py:663-665)
            }
            if (diag) {
                const int jd = octet_diag(o, n);
                if (jd < nvalid) {
                    const float d = diag[jd < n - o.c ? o.r : o.r + 1];
#pragma unroll
                    for (int j = 0; j < 8; ++j) if (j == jd) v[j] = d;
                }
            }
        } else {                                              // one block per row, up to eight rows in the group
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int r = min(((int)e + j) / n, n - 1), c = (int)e + j - r * n;
                const float am = __ldg(absmax + r);
                v[j] = fmaf(code_s[idx[j]], am, am == 0.0f ? 0.0f : -0.0f);
                if (diag && r == c) v[j] = diag[r];
            }
        }
        T *dst = out + e;
        if (vec_out && nvalid == 8) store_vec<T, 8>(dst, v);
        else {
#pragma unroll
            for (int j = 0; j < 8; ++j) if (j < nvalid) dst[j] = from_f32<T>(v[j]);
        }
    }
}

// ------------------------------------------------------------------------------------
// Self-test of the fast division: counts pairs (x, d), d in [2^-40, 2^60], |x| <= d, whose
// reciprocal-based quotient differs in any bit from the IEEE division (quotients below 2^-60
// in magnitude are exempt, as in the quantizer).  Pairs come from a counter-based hash.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned mix32(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull; z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (unsigned)((z ^ (z >> 31)) >> 16);
}
__global__ void k_selftest_division(unsigned long long seed, unsigned long long pairs, unsigned long long *mismatches) {
    unsigned long long bad = 0;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < pairs;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const unsigned a = mix32(seed + 2 * i), b = mix32(seed + 2 * i + 1);
        // d: exponent in [-40, 60), random mantissa; x = d * (fraction in [-1, 1]) with a random small exponent drop
        const int ed = (int)(a % 100u) - 40 + 127;
        const float d = __uint_as_float(((unsigned)ed << 23) | (b & 0x7FFFFFu));
        const unsigned c = mix32(seed ^ (i * 0xD1342543DE82EF95ull));
        const int drop = (c >> 24) % 40;                       // |x| spans 40 binades below d
        float x = __uint_as_float(((unsigned)(ed - drop) << 23) | (c & 0x7FFFFFu));
        if (fabsf(x) > d) x = d;
        if (a & 0x80000000u) x = -x;
        if ((c & 0xFF00u) == 0) x = (c & 1) ? d : -d;           // exact +-1 quotients
        const float q_ref = __fdiv_rn(x, d);
        const float q = div_by_recip(x, d, __frcp_rn(d));
        if (fabsf(q_ref) >= 8.6736174e-19f && __float_as_uint(q) != __float_as_uint(q_ref)) ++bad;   // 2^-60
    }
    if (bad) atomicAdd(mismatches, bad);
}

int launch_selftest_division(unsigned long long seed, unsigned long long pairs, unsigned long long *mismatches_dev,
                             cudaStream_t s) {
    if (!mismatches_dev) return record(QT_ERR_ARG);
    k_selftest_division<<<148 * 8, 256, 0, s>>>(seed, pairs, mismatches_dev);
    count_launch(1);
    return check_launch();
}

// ------------------------------------------------------------------------------------
// Host launchers.
// ------------------------------------------------------------------------------------
static int sm_count() { return device_sm_count(); }

static inline bool aligned(const void *p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// grid.x for `work_items` thread-iterations of one matrix, `count` matrices in grid.y:
// enough CTAs to fill the machine a few times over, at least `min_iters` iterations per
// thread where the matrix is large enough to amortise the per-CTA table build.
static unsigned grid_x_for(long long thread_iters, int count, int min_iters) {
    long long ctas = (thread_iters + (long long)kThreads * min_iters - 1) / ((long long)kThreads * min_iters);
    const long long target = (long long)sm_count() * 8;      // resident CTAs of 256 threads per SM
    long long per_matrix_cap = (target * 4 + count - 1) / count;
    if (per_matrix_cap < 1) per_matrix_cap = 1;
    if (ctas > per_matrix_cap) ctas = per_matrix_cap;
    if (ctas < 1) ctas = 1;
    return (unsigned)ctas;
}

template <typename T, int BITS>
static void launch_quantize_typed(const QuantArgs &a, cudaStream_t s) {
    const int n = a.n, nb = (n + a.bs - 1) / a.bs;
    const T *A = static_cast<const T *>(a.A);
    const size_t esz = sizeof(T);
    const bool many = a.count > 1;
    const bool vec8 = n % 8 == 0 && aligned(A, 16) && aligned(a.out, BITS == 4 ? 4 : 8) &&
                      (!many || ((a.strideA * (long long)esz) % 16 == 0 && a.stride_out % (BITS == 4 ? 4 : 8) == 0));
    int epl = (a.bs <= 256 && vec8) ? 8 : 0;
    // 4-bit, block 64 (the optimizers' configuration): 16 elements per lane, 4 lanes per block
    if (BITS == 4 && a.bs == 64 && epl == 8) epl = 16;
    if (epl) {
        const int lpu = a.bs / epl;
        // every CTA builds the code tables once: exactly one resident wave (or fewer CTAs when the
        // batch is small), striding over the units of the whole batch
        const long long wunits = (long long)((n + 32 / lpu - 1) / (32 / lpu)) * nb;   // warp units per matrix
        if (wunits * a.count >= (1ll << 31) - (1ll << 24) && a.count > 1) {   // warp-unit numbers are 32-bit in the kernel
            const int half = a.count / 2;
            QuantArgs lo = a, hi = a;
            lo.count = half;
            hi.count = a.count - half;
            hi.A = (const char *)a.A + (long long)half * a.strideA * (long long)esz;
            hi.absmax = a.absmax + (long long)half * a.stride_absmax;
            hi.diag = a.diag ? a.diag + (long long)half * a.stride_diag : nullptr;
            hi.out = a.out + (long long)half * a.stride_out;
            launch_quantize_typed<T, BITS>(lo, s);
            launch_quantize_typed<T, BITS>(hi, s);
            return;
        }
        const int resident = 4;                              // the kernels' launch bounds
        // 256-bit loads need every lane's fp32 octets on a 32-byte boundary
        const int wide = (epl == 16 && (esz == 2 || (aligned(A, 32) && (!many || (a.strideA * (long long)esz) % 32 == 0)))) ? 1 : 0;
        long long ctas = (long long)sm_count() * resident;
        const long long needed = (wunits * a.count + kThreads / 32 - 1) / (kThreads / 32);
        if (ctas > needed) ctas = needed;
        if (ctas < 1) ctas = 1;
        dim3 grid((unsigned)ctas);
#define QT_LAUNCH_Q(E, L)                                                                          \
        k_quantize_vec<T, BITS, E, L><<<grid, kThreads, 0, s>>>(A, a.strideA, a.code, n, nb, a.count, a.absmax, \
            a.stride_absmax, a.diag, a.stride_diag, a.out, a.stride_out, wide)
        if constexpr (BITS == 4) { if (epl == 16) { QT_LAUNCH_Q(16, 4); count_launch(1); return; } }
        if (epl == 8 && lpu == 8) QT_LAUNCH_Q(8, 8);
        else if (epl == 8 && lpu == 16) QT_LAUNCH_Q(8, 16);
        else QT_LAUNCH_Q(8, 32);
#undef QT_LAUNCH_Q
        count_launch(1);
        return;
    }
    if (n < 8) {
        k_quantize_tiny<T, BITS><<<a.count, 64, 0, s>>>(A, a.strideA, a.code, n, a.absmax, a.stride_absmax, a.diag, a.stride_diag,
                                                       a.out, a.stride_out);
        count_launch(1);
        return;
    }
    int bs_shift = 0;
    while ((1 << bs_shift) < a.bs) ++bs_shift;
    const int groups = (n + 7) / 8;
    const long long work = (long long)groups * a.count;
    const long long wave = (long long)sm_count() * 4;         // the kernel's launch bounds
    const int vec_in = aligned(A, 16) && (!many || (a.strideA * (long long)esz) % 16 == 0);
    const int vec_out = aligned(a.out, BITS == 4 ? 4 : 8) && (!many || a.stride_out % (BITS == 4 ? 4 : 8) == 0);
    k_quantize_rows<T, BITS><<<(unsigned)(work < wave ? work : wave), kThreads, sizeof(float2) * 8 * nb, s>>>(
        A, a.strideA, a.code, n, nb, bs_shift, groups, a.count, a.absmax, a.stride_absmax, a.diag, a.stride_diag, a.out, a.stride_out,
        vec_in, vec_out);
    count_launch(1);
}

int launch_quantize(const QuantArgs &a, cudaStream_t s) {
    if (a.bits != 4 && a.bits != 8) return record(QT_ERR_BITS);
    if (!valid_blocksize(a.bs)) return record(QT_ERR_BLOCKSIZE);
    if (a.a_dtype != QT_F32 && a.a_dtype != QT_BF16) return record(QT_ERR_DTYPE);
    if (a.n < 0 || a.count < 0 || a.n > 46340 || a.count > 65535) return record(QT_ERR_ARG);
    if (a.n == 0 || a.count == 0) return record(QT_OK);
    if (!a.A || !a.code || !a.absmax || !a.out) return record(QT_ERR_ARG);
    if (!aligned(a.absmax, 4) || !aligned(a.code, 4) || (a.diag && !aligned(a.diag, 4))) return record(QT_ERR_ARG);
    if (!aligned(a.A, a.a_dtype == QT_F32 ? 4 : 2)) return record(QT_ERR_ARG);
    if (a.a_dtype == QT_F32) {
        if (a.bits == 4) launch_quantize_typed<float, 4>(a, s); else launch_quantize_typed<float, 8>(a, s);
    } else {
        if (a.bits == 4) launch_quantize_typed<__nv_bfloat16, 4>(a, s); else launch_quantize_typed<__nv_bfloat16, 8>(a, s);
    }
    return check_launch();
}

template <typename T, int BITS>
static void launch_dequantize_typed(const DequantArgs &a, cudaStream_t s) {
    const int n = a.n, nb = (n + a.bs - 1) / a.bs;
    T *out = static_cast<T *>(a.out);
    const size_t esz = sizeof(T);
    int bs_shift = 0;
    while ((1 << bs_shift) < a.bs) ++bs_shift;
    const bool many = a.count > 1;
    // Eight elements per thread make one store: 256 bits of fp32 or 128 bits of bf16.
    const size_t in_bytes = BITS == 4 ? 4 : 8, out_bytes = esz == 4 ? 32 : 16;
    const int vec_in = aligned(a.A, in_bytes) && (!many || a.strideA % (long long)in_bytes == 0);
    const int vec_out = aligned(out, out_bytes) && (!many || (a.stride_out * (long long)esz) % (long long)out_bytes == 0);
    const long long chunks = ((long long)n * n + 7) / 8;
    dim3 grid(grid_x_for(chunks, a.count, 4), a.count);
    if (n % 8 == 0 && vec_in && vec_out)
        k_dequantize_vec<T, BITS, 8><<<grid, kThreads, 0, s>>>(a.A, a.strideA, a.code, n, nb, bs_shift, a.absmax,
            a.stride_absmax, a.diag, a.stride_diag, out, a.stride_out);
    else
        k_dequantize_flat<T, BITS><<<grid, kThreads, 0, s>>>(a.A, a.strideA, a.code, n, nb, bs_shift, a.absmax,
            a.stride_absmax, a.diag, a.stride_diag, out, a.stride_out, vec_in, vec_out);
    count_launch(1);
}

int launch_dequantize(const DequantArgs &a, cudaStream_t s) {
    if (a.bits != 4 && a.bits != 8) return record(QT_ERR_BITS);
    if (!valid_blocksize(a.bs)) return record(QT_ERR_BLOCKSIZE);
    if (a.out_dtype != QT_F32 && a.out_dtype != QT_BF16) return record(QT_ERR_DTYPE);
    if (a.n < 0 || a.count < 0 || a.n > 46340 || a.count > 65535) return record(QT_ERR_ARG);
    if (a.n == 0 || a.count == 0) return record(QT_OK);
    if (!a.A || !a.code || !a.absmax || !a.out) return record(QT_ERR_ARG);
    if (!aligned(a.absmax, 4) || !aligned(a.code, 4) || (a.diag && !aligned(a.diag, 4))) return record(QT_ERR_ARG);
    if (!aligned(a.out, a.out_dtype == QT_F32 ? 4 : 2)) return record(QT_ERR_ARG);
    if (a.out_dtype == QT_F32) {
        if (a.bits == 4) launch_dequantize_typed<float, 4>(a, s); else launch_dequantize_typed<float, 8>(a, s);
    } else {
        if (a.bits == 4) launch_dequantize_typed<__nv_bfloat16, 4>(a, s); else launch_dequantize_typed<__nv_bfloat16, 8>(a, s);
    }
    return check_launch();
}

int launch_state_exponents(const float *absmax, long long stride_absmax, int n_absmax, const float *diag, long long stride_diag,
                           int n_diag, const int *slots, int count, int target, int *exp_out, cudaStream_t s) {
    if (count < 0 || n_absmax < 0 || !absmax || !exp_out) return record(QT_ERR_ARG);
    if (count == 0) return record(QT_OK);
    k_state_amax<<<count, 256, 0, s>>>(absmax, stride_absmax, n_absmax, diag, stride_diag, n_diag, slots, nullptr, exp_out, target);
    count_launch(1);
    return check_launch();
}

int launch_dequantize_planes(const DequantArgs &a, const int *slots, void *hi, void *lo, long long ldp, long long strideP,
                             cudaStream_t s, float *amax_scratch, int target, int *exp_out) {
    if (a.bits != 4 && a.bits != 8) return record(QT_ERR_BITS);
    if (!valid_blocksize(a.bs)) return record(QT_ERR_BLOCKSIZE);
    if (a.n < 0 || a.count < 0 || a.n > 46340 || a.count > 65535) return record(QT_ERR_ARG);
    if (a.n == 0 || a.count == 0) return record(QT_OK);
    if (!a.A || !a.code || !a.absmax || !hi || !lo) return record(QT_ERR_ARG);
    // eight elements per thread: 16-byte plane stores, 4/8-byte code loads
    if (a.n % 8 || ldp % 8 || strideP % 8 || !aligned(hi, 16) || !aligned(lo, 16) || ldp < a.n) return record(QT_ERR_UNSUPPORTED);
    const int in_bytes = a.bits == 4 ? 4 : 8;
    if (!aligned(a.A, in_bytes) || a.strideA % in_bytes) return record(QT_ERR_UNSUPPORTED);
    if (!aligned(a.absmax, 4) || !aligned(a.code, 4) || (a.diag && !aligned(a.diag, 4))) return record(QT_ERR_ARG);
    const int n = a.n, nb = (n + a.bs - 1) / a.bs;
    int bs_shift = 0;
    while ((1 << bs_shift) < a.bs) ++bs_shift;
    // 16 elements per thread: 256-bit plane stores (32-byte rows) and 8/16-byte code loads
    const int in16 = a.bits == 4 ? 8 : 16;
    const bool wide = n % 16 == 0 && ldp % 16 == 0 && strideP % 16 == 0 && aligned(hi, 32) && aligned(lo, 32) &&
                      aligned(a.A, in16) && a.strideA % in16 == 0 && a.bs >= 16;
    dim3 grid(grid_x_for((long long)n * (n / (wide ? 16 : 8)), a.count, 4), a.count);
    const bool f16 = amax_scratch != nullptr;
    if (f16) {
        k_state_amax<<<a.count, 256, 0, s>>>(a.absmax, a.stride_absmax, n * nb, a.diag, a.stride_diag, n, slots, amax_scratch);
        count_launch(1);
    }
#define QT_DQP(B, E, H)                                                                                                 \
    k_dequantize_planes<B, E, H><<<grid, kThreads, 0, s>>>(a.A, a.strideA, a.code, n, nb, bs_shift, a.absmax, a.stride_absmax, \
        a.diag, a.stride_diag, slots, static_cast<__nv_bfloat16 *>(hi), static_cast<__nv_bfloat16 *>(lo), ldp, strideP,   \
        amax_scratch, target, exp_out)
    if (f16) {
        if (a.bits == 4) { if (wide) QT_DQP(4, 16, true); else QT_DQP(4, 8, true); }
        else { if (wide) QT_DQP(8, 16, true); else QT_DQP(8, 8, true); }
    } else {
        if (a.bits == 4) { if (wide) QT_DQP(4, 16, false); else QT_DQP(4, 8, false); }
        else { if (wide) QT_DQP(8, 16, false); else QT_DQP(8, 8, false); }
    }
#undef QT_DQP
    count_launch(1);
    return check_launch();
}

}  // namespace qt
