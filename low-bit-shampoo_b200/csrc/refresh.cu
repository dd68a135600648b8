// Refresh of one order class as one host call: statistics L <- w1 V^T diag(S) V + w2 G G^T, eigenbasis by one subspace
// step (QR of L V), Rayleigh quotients, kept half of the spectrum, and the inverse root from it (reference project paths
// optimizers/shampoo2.py:169-232, qtensor/utils.py:156-227, qtensor/functional.py:749-762).
//
// Everything is batched over the class and runs in a workspace of the caller; nothing is read back.  A class of order
// 1000 is some 110 launches in a chain; issued from Python, one call each with its own allocations, the chain was bound by
// the host (16 us per launch, 6.2 ms for two classes of eight matrices of 512 and 1000).  Intermediate results stay in
// the form the next product reads: the dequantizer, the panel kernels, the merge of T and the product epilogues write operand
// planes, epilogues take the magnitudes that planes are scaled by, and symmetric products compute half their tiles.
#include "quant_device.cuh"
#include "gemm_api.cuh"
#include "tc_device.cuh"
#include <cuda_fp16.h>

namespace qt {

static constexpr int kTarget = 9;                 // freshly split planes: largest scaled entry below 2^9
static constexpr int kMaxExp = 15;                // plane results are placed below 2^15
static constexpr int kBasisExp = kTarget - 1;     // entries of orthonormal rows and of Householder vectors: at most 2
static constexpr int kLooseExp = kTarget - 3;     // entries of a rectified basis: at most 8 (with a wide margin)
static constexpr int kThreadsR = 256;

__device__ __forceinline__ void put_f16_pair(__half *hi, __half *lo, const float (&v)[16]) {
    unsigned H[8], L[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const __half h0 = __float2half_rn(v[2 * j]), h1 = __float2half_rn(v[2 * j + 1]);
        const __half l0 = __float2half_rn(v[2 * j] - __half2float(h0)), l1 = __float2half_rn(v[2 * j + 1] - __half2float(h1));
        H[j] = (unsigned)__half_as_ushort(h0) | ((unsigned)__half_as_ushort(h1) << 16);
        L[j] = (unsigned)__half_as_ushort(l0) | ((unsigned)__half_as_ushort(l1) << 16);
    }
    stg256u(reinterpret_cast<unsigned *>(hi), H);
    stg256u(reinterpret_cast<unsigned *>(lo), L);
}

// Rows of stored eigenbases (all, or those of an index list) dequantized to fp32 and, in the same pass, to planes of
// fixed exponent.  Sixteen columns per thread; see k_apply_planes for codes that start at any nibble.
template <int BITS>
__global__ void __launch_bounds__(kThreadsR)
k_basis_rows(const unsigned char *__restrict__ codes, long long stride_codes, const float *__restrict__ absmax_base, long long stride_absmax,
             const float *__restrict__ code, int n, int nb, int bs_shift, const long long *__restrict__ index, long long stride_index, int rows,
             float *__restrict__ X, long long ldx, long long strideX, __half *__restrict__ hi, __half *__restrict__ lo, long long ldp, long long strideP, float scale) {
    chain_wait();
    __shared__ float2 pair_lut[BITS == 4 ? 256 : 1];
    __shared__ float code_s[BITS == 8 ? 256 : 1];
    if constexpr (BITS == 4) pair_lut[threadIdx.x] = make_float2(__ldg(code + (threadIdx.x >> 4)), __ldg(code + (threadIdx.x & 15)));
    else code_s[threadIdx.x] = __ldg(code + threadIdx.x);
    __syncthreads();
    const int m = blockIdx.y;
    const unsigned char *in = codes + (long long)m * stride_codes;
    const float *absmax = absmax_base + (long long)m * stride_absmax;
    const long long *idx = index ? index + (long long)m * stride_index : nullptr;
    float *x = X + (long long)m * strideX;
    hi += (long long)m * strideP;
    lo += (long long)m * strideP;
    const int c16 = (n + 15) >> 4, total = rows * c16;
    const bool even = n % 16 == 0, wide = ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(X) & 31) == 0 && strideX % 8 == 0;
    const unsigned last_word = ((unsigned)n * (unsigned)n - 1u) >> 3;
    for (int t = blockIdx.x * kThreadsR + threadIdx.x; t < total; t += gridDim.x * kThreadsR) {
        const int rr = t / c16, c = (t - rr * c16) * 16;
        const int r = idx ? (int)idx[rr] : rr;
        const unsigned f = (unsigned)r * (unsigned)n + (unsigned)c;
        const float am = __ldg(absmax + (long long)r * nb + (c >> bs_shift));
        const float z = (am == 0.0f) ? 0.0f : -0.0f;
        float v[16];
        if constexpr (BITS == 4) {
            unsigned w0, w1;
            if (even) {
                const uint2 ww = __ldg(reinterpret_cast<const uint2 *>(in + (f >> 1)));
                w0 = __byte_perm(ww.x, 0, 0x0123); w1 = __byte_perm(ww.y, 0, 0x0123);
            } else {
                const unsigned *wp = reinterpret_cast<const unsigned *>(in);
                const unsigned i = f >> 3, sh = (f & 7u) * 4u;
                const unsigned x0 = __byte_perm(__ldg(wp + i), 0, 0x0123);
                const unsigned x1 = i + 1 <= last_word ? __byte_perm(__ldg(wp + i + 1), 0, 0x0123) : 0u;
                const unsigned x2 = i + 2 <= last_word ? __byte_perm(__ldg(wp + i + 2), 0, 0x0123) : 0u;
                w0 = __funnelshift_l(x1, x0, sh); w1 = __funnelshift_l(x2, x1, sh);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float2 p = pair_lut[((j < 4 ? w0 : w1) >> (24 - 8 * (j & 3))) & 255u];
                v[2 * j] = fmaf(p.x, am, z);
                v[2 * j + 1] = fmaf(p.y, am, z);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = c + j < n ? fmaf(code_s[__ldg(in + f + j)], am, z) : 0.0f;
        }
        float *xr = x + (long long)rr * ldx + c;
        if (wide && c + 16 <= n) { stg256f(xr, v); stg256f(xr + 8, v + 8); }
        else {
#pragma unroll
            for (int j = 0; j < 16; ++j) if (c + j < n) xr[j] = v[j];
        }
        float worst = 0.0f;
#pragma unroll
        for (int j = 0; j < 16; ++j) { v[j] = fminf(fmaxf(v[j] * scale, -65000.0f), 65000.0f); worst = fmaxf(worst, c + j < n ? fabsf(v[j]) : 0.0f); }
        if (worst >= 65000.0f) atomicCAS(&g_gemm_error, 0, QT_ERR_RANGE);
        put_f16_pair(hi + rr * ldp + c, lo + rr * ldp + c, v);
    }
}

// fp32 rows (gathered by an index list, scaled) -> planes.  Scratch matrices and planes have rows of a multiple of 32 bytes, so a
// thread takes eight columns: one 256-bit load, one 128-bit store per plane; what stands behind a ragged row is read and
// written as zeros into the planes' padding.  Bound by HBM: 124 x 768^2 floats 181 -> 97 us (6.0 TB/s; two columns a thread
// before, which kept too few bytes in flight).  `b` (with b.hi): the same rows once more, scaled by its own factors.
// Exponent: exponent_for(amax[m], target) if amax, else the constant `exp0`.
struct RowPlanes { __half *hi, *lo; const float *scale, *amax; int *exp_out; int exp0; };
__global__ void __launch_bounds__(kThreadsR)
k_rows_to_planes(const float *__restrict__ X, long long ldx, long long strideX, int rows, int cols, const long long *__restrict__ index,
                 long long stride_index, long long stride_scale, long long ldp, long long strideP, const RowPlanes a, const RowPlanes b, int target) {
    chain_wait();
    const int m = blockIdx.y;
    const float *x = X + (long long)m * strideX;
    const long long *idx = index ? index + (long long)m * stride_index : nullptr;
    const bool two = b.hi != nullptr;
    const int ea = a.amax ? exponent_for(a.amax[m], target) : a.exp0, eb = two ? (b.amax ? exponent_for(b.amax[m], target) : b.exp0) : 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (a.exp_out) a.exp_out[m] = ea;
        if (two && b.exp_out) b.exp_out[m] = eb;
    }
    const float sa = exp2f((float)ea), sb = exp2f((float)eb);
    const int c8 = (cols + 7) >> 3, total = rows * c8;
    float worst = 0.0f;
#pragma unroll 2
    for (int t = blockIdx.x * kThreadsR + threadIdx.x; t < total; t += gridDim.x * kThreadsR) {
        const int r = t / c8, c = (t - r * c8) * 8;
        float v[8];
        ldg256f(x + (idx ? idx[r] : (long long)r) * ldx + c, v);
        if (c + 8 > cols) {
#pragma unroll
            for (int q = 0; q < 8; ++q) if (c + q >= cols) v[q] = 0.0f;
        }
        auto put = [&](const RowPlanes &o, float s) {
            const float f = o.scale ? o.scale[(long long)m * stride_scale + r] * s : s;
            unsigned h[4], l[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float x0 = fminf(fmaxf(v[2 * q] * f, -65000.0f), 65000.0f), x1 = fminf(fmaxf(v[2 * q + 1] * f, -65000.0f), 65000.0f);
                worst = fmaxf(worst, fmaxf(fabsf(x0), fabsf(x1)));
                const __half2 hh = __floats2half2_rn(x0, x1);
                const float2 hf = __half22float2(hh);
                const __half2 ll = __floats2half2_rn(x0 - hf.x, x1 - hf.y);
                h[q] = *reinterpret_cast<const unsigned *>(&hh);
                l[q] = *reinterpret_cast<const unsigned *>(&ll);
            }
            const long long at = (long long)m * strideP + (long long)r * ldp + c;
            *reinterpret_cast<uint4 *>(o.hi + at) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4 *>(o.lo + at) = make_uint4(l[0], l[1], l[2], l[3]);
        };
        put(a, sa);
        if (two) put(b, sb);
    }
    if (worst >= 65000.0f) atomicCAS(&g_gemm_error, 0, QT_ERR_RANGE);
}

// Q = I, fp32 and planes.
__global__ void __launch_bounds__(kThreadsR)
k_identity(float *__restrict__ X, long long ldx, __half *__restrict__ hi, __half *__restrict__ lo, int n, long long ldp, long long strideP, float scale) {
    chain_wait();
    float *x = X + (long long)blockIdx.y * n * ldx;
    hi += (long long)blockIdx.y * strideP;
    lo += (long long)blockIdx.y * strideP;
    const __half one = __float2half_rn(scale), zero = __float2half_rn(0.0f);
    const int c2 = (int)ldp >> 1, total = n * c2;
    for (int t = blockIdx.x * kThreadsR + threadIdx.x; t < total; t += gridDim.x * kThreadsR) {
        const int r = t / c2, c = (t - r * c2) * 2;
        if (c < n) x[(long long)r * ldx + c] = r == c ? 1.0f : 0.0f;
        if (c + 1 < n) x[(long long)r * ldx + c + 1] = r == c + 1 ? 1.0f : 0.0f;
        *reinterpret_cast<__half2 *>(hi + (long long)r * ldp + c) = __halves2half2(r == c ? one : zero, r == c + 1 ? one : zero);
        *reinterpret_cast<__half2 *>(lo + (long long)r * ldp + c) = __halves2half2(zero, zero);
    }
}

// Kept half of the spectrum of every matrix: Rayleigh quotients from the products' partial sums (added in a fixed
// order), sorted ascending with their row numbers - ties by row number - in shared memory (n <= 2048).
__global__ void __launch_bounds__(1024)
k_spectrum(const float *__restrict__ part, int parts, int n, int keep, float *__restrict__ S, long long *__restrict__ keep_idx, float *__restrict__ max_eig) {
    chain_wait();
    extern __shared__ unsigned long long keys[];
    const int m = blockIdx.x;
    int size = 2;
    while (size < n) size <<= 1;
    const float *p = part + (long long)m * parts * n;
    for (int i = threadIdx.x; i < size; i += blockDim.x) {
        unsigned long long key = ~0ull;
        if (i < n) {
            float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            for (int q = 0; q < parts; ++q) a[q & 3] += __ldg(p + (long long)q * n + i);
            const unsigned u = __float_as_uint((a[0] + a[1]) + (a[2] + a[3]));
            const unsigned ord = (u & 0x80000000u) ? ~u : (u | 0x80000000u);   // orders like the values, NaN last
            key = ((unsigned long long)ord << 32) | (unsigned)i;
        }
        keys[i] = key;
    }
    for (int k = 2; k <= size; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            __syncthreads();
            for (int i = threadIdx.x; i < size; i += blockDim.x) {
                const int o = i ^ j;
                if (o > i) {
                    const unsigned long long a = keys[i], b = keys[o];
                    if ((a > b) == ((i & k) == 0)) { keys[i] = b; keys[o] = a; }
                }
            }
        }
    __syncthreads();
    auto value = [&](int i) {
        const unsigned ord = (unsigned)(keys[i] >> 32);
        return __uint_as_float((ord & 0x80000000u) ? (ord & 0x7fffffffu) : ~ord);
    };
    for (int i = threadIdx.x; i < keep; i += blockDim.x) {
        S[(long long)m * keep + i] = value(i);
        keep_idx[(long long)m * keep + i] = (long long)(unsigned)keys[i];
    }
    if (threadIdx.x == 0) max_eig[m] = value(n - 1);
}

// Row weights of a class and the bound on the scaled rows that its planes are placed by.  eps < 0: the kept eigenvalues
// themselves; else (S + eps lambda_max)^(-1/p), where a quotient at or below -rho counts as zero
// (qtensor/functional.py:760-762; see ridged_inverse_root in this package's qtensor/functional.py).
__global__ void __launch_bounds__(256)
k_row_weights(const float *__restrict__ S, const float *__restrict__ max_eig, int keep, float eps, float inv_p, float basis_bound,
              float *__restrict__ weights, float *__restrict__ bound) {
    chain_wait();
    __shared__ float red[8];
    const int m = blockIdx.x;
    const float rho = eps >= 0.0f ? eps * max_eig[m] : 0.0f;
    float am = 0.0f;
    for (int i = threadIdx.x; i < keep; i += blockDim.x) {
        float w = S[(long long)m * keep + i];
        if (eps >= 0.0f) {
            const float t = w + rho;
            w = 1.0f / powf(t > 0.0f ? t : rho, inv_p);
        }
        weights[(long long)m * keep + i] = w;
        am = fmaxf(am, fabsf(w));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, off));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = am;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i) am = fmaxf(am, red[i]);
        bound[m] = am * basis_bound;
    }
}

// Codes of Q^T (4 bits, block 64, n a multiple of 16) from Q row-major: a CTA stages 64 rows x 64 columns of Q and
// quantizes its columns, so that the transposed fp32 copy (8 bytes per element written and read) does not exist.  Four
// lanes per block as in k_quantize_vec, same arithmetic.
__global__ void __launch_bounds__(256)
k_quantize_transposed(const float *__restrict__ Q, long long ldq, long long strideQ, const float *__restrict__ code, int n, int nb,
                      float *__restrict__ absmax_base, long long stride_absmax, unsigned char *__restrict__ out_base, long long stride_out) {
    chain_wait();
    __shared__ CodeTables<16> tab;
    __shared__ float tile[64][65];
    build_tables<16>(tab, code);
    const bool lean_launch = !tab.lut_bad && !tab.need_clamp && tab.perm_identity && !tab.tiny_thr;
    const int tiles = nb * nb, m = blockIdx.y;
    const float *q = Q + (long long)m * strideQ;
    for (int tt = blockIdx.x; tt < tiles; tt += gridDim.x) {
        const int k0 = (tt / nb) * 64, r0 = (tt % nb) * 64;   // rows k0.. and columns r0.. of Q: block k0 / 64 of the rows r0.. of Q^T
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int r = (threadIdx.x >> 6) + 4 * i, c = threadIdx.x & 63;
            tile[r][c] = (k0 + r < n && r0 + c < n) ? __ldg(q + (long long)(k0 + r) * ldq + r0 + c) : 0.0f;
        }
        __syncthreads();
        const int row = threadIdx.x >> 2, part = threadIdx.x & 3;   // row r0 + row of Q^T, elements k0 + 16 part ..
        float x[16], amax = 0.0f;
#pragma unroll
        for (int j = 0; j < 16; ++j) { x[j] = tile[16 * part + j][row]; amax = fmaxf(amax, fabsf(x[j])); }
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        if (r0 + row >= n) continue;
        if (part == 0) absmax_base[(long long)m * stride_absmax + (long long)(r0 + row) * nb + k0 / 64] = amax;
        if (k0 + 16 * part >= n) continue;
        unsigned w0 = 0, w1 = 0;
        bool generic = !(lean_launch && ((amax >= 9.094947e-13f && amax <= 1.1529215e18f) || amax == 0.0f));
        if (!generic && amax != 0.0f) {
            const float rcp = __frcp_rz(amax);
            unsigned w[16], nearest = 0xffffffffu;
#pragma unroll
            for (int j = 0; j < 16; ++j) { w[j] = code_word(tab, tab.lut_shift, tab.lut_mask, x[j], rcp); nearest = min(nearest, w[j] & 0xffffffu); }
            w0 = pack_codes(w);
            w1 = pack_codes(w + 8);
            generic = nearest <= 8u;
        }
        if (generic) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                LaneVals<8> xv;
#pragma unroll
                for (int j = 0; j < 8; ++j) xv.v[j] = x[8 * h + j];
                const unsigned long long pk = quantize_lane_generic<16, 8>(tab, xv, amax);
                unsigned w[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) w[j] = (unsigned)(pk >> (8 * j)) << 24;
                (h == 0 ? w0 : w1) = pack_codes(w);
            }
        }
        const long long e = (long long)(r0 + row) * n + k0 + 16 * part;
        *reinterpret_cast<uint2 *>(out_base + (long long)m * stride_out + (e >> 1)) = make_uint2(w0, w1);
    }
}

__global__ void __launch_bounds__(256)
k_transpose(const float *__restrict__ X, long long ldx, float *__restrict__ Y, int n) {
    chain_wait();
    __shared__ float t[32][33];
    const long long o = (long long)blockIdx.z * n * n, ox = (long long)blockIdx.z * n * ldx;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    for (int i = ty; i < 32; i += 8) if (r0 + i < n && c0 + tx < n) t[i][tx] = X[ox + (long long)(r0 + i) * ldx + c0 + tx];
    __syncthreads();
    for (int i = ty; i < 32; i += 8) if (c0 + i < n && r0 + tx < n) Y[o + (long long)(c0 + i) * n + r0 + tx] = t[tx][i];
}

// ------------------------------------------------------------------------------------
// Host side.
// ------------------------------------------------------------------------------------
static inline long long up(long long x, long long q) { return (x + q - 1) / q * q; }
static inline int ceil_log2(long long x) { int k = 0; while ((1ll << k) < x) ++k; return k; }

// A batch of matrices as scaled fp16 planes; `exp` per matrix (null: exp0 alone), entries below 2^tmax.
struct P2 {
    __half *hi, *lo; long long ld, stride; int *exp; int exp0, tmax;
    P2 window(long long r, long long c) const { P2 w = *this; w.hi += r * ld + c; w.lo += r * ld + c; return w; }
};

struct Bump {
    char *base; size_t used, size;
    void *take(size_t bytes) {
        const size_t at = (used + 255) & ~(size_t)255;
        used = at + bytes;
        return base ? base + at : nullptr;
    }
    template <class T> T *of(long long n) { return static_cast<T *>(take((size_t)n * sizeof(T))); }
    P2 planes(int m, long long rows, long long cols, int exp0, int *exp = nullptr) {
        P2 p;
        p.ld = up(cols, 16); p.stride = rows * p.ld; p.exp = exp; p.exp0 = exp0; p.tmax = kTarget;
        p.hi = of<__half>(m * p.stride); p.lo = of<__half>(m * p.stride);
        return p;
    }
};

// alpha op(A) op(B) + beta C: into D and / or the planes P (exponents as P says; `rel`: worst-case exponents, written to P.exp).
struct Out { float *D = nullptr; long long ldd = 0, strideD = 0; const P2 *P = nullptr; bool rel = false; const float *C = nullptr; float alpha = 1.0f, beta = 0.0f;
             int sym = 0; float *amax = nullptr; const int *slot = nullptr; float *cd = nullptr; };
// The stream of a pass.  In a small class the next kernel is brought onto the chip while its predecessor ends (see
// launch_chained): some 150 launches of 10 to 60 us follow each other, and start-up and prologue are 2 us of each (8
// matrices of 1000 and 8 of 512: 3.55 -> 3.35 ms, 4 of 1189 and 4 of 777: 3.90 -> 3.70).  Where a product has several
// rounds of tiles the kernels are long, and waiting ones hold SMs that other classes would use (ViT-B/32: 24.3 -> 24.8 ms).
struct Queue {
    cudaStream_t stream;
    bool chained;
    operator cudaStream_t() const { return stream; }
};

static int product(const P2 &A, bool ta, const P2 &B, bool tb, int M, int N, int K, int batch, const Out &o, const Queue &s) {
    GemmArgs a{A.hi, A.lo, A.ld, A.stride, ta ? 1 : 0, B.hi, B.lo, B.ld, B.stride, tb ? 0 : 1, M, N, K, batch, o.alpha, o.beta,
               o.C, o.ldd, o.strideD, o.D, o.ldd, o.strideD, o.P ? o.P->hi : nullptr, o.P ? o.P->lo : nullptr, o.P ? o.P->ld : 0, o.P ? o.P->stride : 0};
    GemmExtras x;
    x.f16 = 1; x.kc = 2; x.a_exp = A.exp; x.b_exp = B.exp; x.ab_exp0 = A.exp0 + B.exp0;
    x.sym = o.sym; x.amax_out = o.amax; x.cd_part = o.cd;
    x.chained = s.chained;                                    // a product is never the first launch of a pass
    if (o.slot) { x.d_slot = o.slot; x.c_follows_d = 1; }
    if (o.P) {
        if (o.rel) { x.out_rel = 1; x.out_exp0 = kMaxExp - ceil_log2(K) - A.tmax - B.tmax; x.out_exp_w = o.P->exp; }
        else { x.out_exp = o.P->exp; x.out_exp0 = o.P->exp0; }
    }
    return launch_gemm_planes(a, nullptr, nullptr, s, nullptr, &x);
}

static dim3 rows_grid(long long threads, int m) {
    long long ctas = (threads + kThreadsR * 2 - 1) / (kThreadsR * 2);
    const long long cap = ((long long)device_sm_count() * 16 + m - 1) / m;
    if (ctas > cap) ctas = cap;
    return dim3((unsigned)(ctas < 1 ? 1 : ctas), (unsigned)m);
}

static int to_planes(const float *X, long long ldx, long long strideX, int rows, int cols, int m, const long long *index, long long stride_index,
                     long long stride_scale, const P2 &a, const float *scale_a, const float *amax_a, const P2 *b, const float *scale_b,
                     const float *amax_b, const Queue &s) {
    RowPlanes ra{a.hi, a.lo, scale_a, amax_a, amax_a ? a.exp : nullptr, a.exp0}, rb{nullptr, nullptr, nullptr, nullptr, nullptr, 0};
    if (b) rb = RowPlanes{b->hi, b->lo, scale_b, amax_b, amax_b ? b->exp : nullptr, b->exp0};
    if (launch_chained(k_rows_to_planes, rows_grid((long long)rows * ((cols + 7) / 8), m), kThreadsR, 0, s, s.chained, X, ldx, strideX, rows, cols, index, stride_index, stride_scale,
                       a.ld, a.stride, ra, rb, kTarget) != cudaSuccess) { cudaGetLastError(); return record(QT_ERR_LAUNCH); }
    count_launch(1);
    return check_launch();
}

static int basis_rows(const qt_refresh_desc &d, int a, int m, const long long *index, int rows, float *X, long long ldx, const P2 &p, const Queue &s, bool first) {
    int shift = 0;
    while ((1 << shift) < d.blocksize) ++shift;
    const int nb = (d.n + d.blocksize - 1) / d.blocksize;
    const unsigned char *codes = d.stat_codes + (long long)a * d.stride_codes;
    const float *absmax = d.stat_absmax + (long long)a * d.n * nb;
    const dim3 grid = rows_grid((long long)rows * ((d.n + 15) / 16), m);
    const float scale = ldexpf(1.0f, kBasisExp);
    auto k = d.bits == 4 ? k_basis_rows<4> : k_basis_rows<8>;
    if (launch_chained(k, grid, kThreadsR, 0, s, s.chained && !first, codes, d.stride_codes, absmax, (long long)d.n * nb, d.code, d.n, nb, shift, index, d.keep, rows, X, ldx, rows * ldx,
                                 p.hi, p.lo, p.ld, p.stride, scale) != cudaSuccess) { cudaGetLastError(); return record(QT_ERR_LAUNCH); }
    count_launch(1);
    return check_launch();
}

#define QT_TRY(expr) do { const int rc_ = (expr); if (rc_ != QT_OK) return rc_; } while (0)

// Q of the QR factorisation of X (m matrices of order n; X and its planes are overwritten): two-level blocked compact-WY
// Householder, LAPACK's sign conventions, as optimizers/_qr.py describes.  Q and its planes stay in step.
struct QrSpace { long long ld; float *V, *T, *G; P2 Pv, Pt, Py, Pw; };
static constexpr int kOuter = 128, kPan = 32;
static void qr_space(Bump &w, int m, int n, QrSpace &q) {
    const int npan = (n + kPan - 1) / kPan, nblk = (n + kOuter - 1) / kOuter;
    q.ld = up(n, 8);
    q.V = w.of<float>((long long)m * n * q.ld);
    q.T = w.of<float>((long long)m * npan * kPan * kPan);
    q.G = w.of<float>((long long)m * kOuter * kOuter);
    q.Pv = w.planes(m * nblk, n, kOuter, kBasisExp);          // one buffer per outer block
    q.Pt = w.planes(m * nblk, kOuter, kOuter, 0, w.of<int>((long long)m * nblk));
    q.Py = w.planes(m, n, kOuter, 0, w.of<int>(m));
    q.Pw = w.planes(m, kOuter, n, 0, w.of<int>(m));
    q.Py.tmax = q.Pw.tmax = kMaxExp;
}
static int qr_batch(int m, int n, float *X, const P2 &Px, float *Q, const P2 &Pq, QrSpace &q, const Queue &s) {
    const long long ld = q.ld, nn = n * ld;                   // fp32 matrices have rows of a multiple of 32 bytes
    const int npan = (n + kPan - 1) / kPan;
    auto block = [&](int J0, P2 &pv, P2 &pt) {
        const int k = J0 / kOuter, wo = n - J0 < kOuter ? n - J0 : kOuter;
        pv = q.Pv; pt = q.Pt;
        pv.hi += (long long)k * m * q.Pv.stride; pv.lo += (long long)k * m * q.Pv.stride;
        pv.ld = up(wo, 16); pv.stride = (long long)(n - J0) * pv.ld;
        pt.hi += (long long)k * m * q.Pt.stride; pt.lo += (long long)k * m * q.Pt.stride;
        pt.ld = up(wo, 16); pt.stride = (long long)wo * pt.ld; pt.exp += (long long)k * m;
        return wo;
    };
    auto reflect = [&](const P2 &pv, const P2 &pt, bool transpose_t, int wo, int rows, int cols, float *target, const P2 &planes) {
        P2 y = q.Py, wp = q.Pw;                               // target <- target - (V T') (V^T target)
        y.ld = up(wo, 16); y.stride = (long long)rows * y.ld;
        wp.ld = up(cols, 16); wp.stride = (long long)wo * wp.ld;
        Out oy; oy.P = &y; oy.rel = true;
        QT_TRY(product(pv, false, pt, transpose_t, rows, wo, wo, m, oy, s));
        Out ow; ow.P = &wp; ow.rel = true;
        QT_TRY(product(pv, true, planes, false, wo, cols, rows, m, ow, s));
        Out o; o.D = target; o.C = target; o.ldd = ld; o.strideD = nn; o.P = &planes; o.alpha = -1.0f; o.beta = 1.0f;
        return product(y, false, wp, false, rows, cols, wo, m, o, s);
    };
    P2 pv, pt;
    for (int J0 = 0; J0 < n; J0 += kOuter) {
        const int wo = block(J0, pv, pt);
        for (int j0 = J0; j0 < J0 + wo; j0 += kPan) {
            const int w = J0 + wo - j0 < kPan ? J0 + wo - j0 : kPan, k = j0 / kPan, prev = j0 > J0 ? kPan : 0;
            QT_TRY(launch_householder_panel(X, nn, n, (int)ld, m, j0, w, q.V, nn, q.T + (long long)k * kPan * kPan, (long long)npan * kPan * kPan, s,
                                            prev, prev ? q.T + (long long)(k - 1) * kPan * kPan : nullptr, J0 + wo,
                                            pv.hi, pv.lo, pv.ld, pv.stride, j0 - J0, j0 - J0, kBasisExp, s.chained));
        }
        Out og; og.D = q.G; og.ldd = wo; og.strideD = (long long)wo * wo; og.sym = 1;
        QT_TRY(product(pv, true, pv, false, wo, wo, n - J0, m, og, s));
        QT_TRY(launch_merge_t(q.G, wo, (long long)wo * wo, q.T + (long long)(J0 / kPan) * kPan * kPan, (long long)npan * kPan * kPan, wo, m, nullptr, 0, s,
                              pt.hi, pt.lo, pt.ld, pt.stride, pt.exp, kTarget, s.chained));
        const int rows = n - J0, t = rows - wo;
        if (t > 0) QT_TRY(reflect(pv, pt, true, wo, rows, t, X + J0 * ld + J0 + wo, Px.window(J0, J0 + wo)));
    }
    if (launch_chained(k_identity, rows_grid((long long)n * (Pq.ld / 2), m), kThreadsR, 0, s, s.chained, Q, ld, Pq.hi, Pq.lo, n, Pq.ld, Pq.stride,
                       ldexpf(1.0f, kBasisExp)) != cudaSuccess) { cudaGetLastError(); return record(QT_ERR_LAUNCH); }
    count_launch(1);
    for (int J0 = (n - 1) / kOuter * kOuter; J0 >= 0; J0 -= kOuter) {
        const int wo = block(J0, pv, pt), rows = n - J0;
        QT_TRY(reflect(pv, pt, false, wo, rows, rows, Q + J0 * ld + J0, Pq.window(J0, J0)));
    }
    return check_launch();
}

// One pass over matrices a .. a+m-1 of the class; with w.base == nullptr only the workspace is measured.
static int refresh_pass(const qt_refresh_desc &d, int a, int m, Bump &w, bool run, cudaStream_t stream) {
    const int n = d.n, keep = d.keep, nb = (n + d.blocksize - 1) / d.blocksize;
    const long long ld = up(n, 8), nn = n * ld;               // fp32 scratch matrices have rows of a multiple of 32 bytes
    const int tiles = (n + 127) / 128;
    const Queue s{stream, (long long)tiles * tiles * m <= 4LL * device_sm_count()};
    float *weights = w.of<float>((long long)m * keep), *bound = w.of<float>(m), *amax = w.of<float>(2 * m);
    int *exps = w.of<int>(4 * m);
    float *S = d.S + (long long)a * keep, *max_eig = d.max_eig + a;
    long long *keep_idx = d.keep_idx + (long long)a * keep;
    unsigned char *codes = const_cast<unsigned char *>(d.stat_codes) + (long long)a * d.stride_codes;
    float *absmax = const_cast<float *>(d.stat_absmax) + (long long)a * n * nb;
    const size_t mark = w.used;
    size_t most = mark;
    if (d.do_stat) {
        // buffers by lifetime: a later result takes the place of one that is no longer read
        float *f1 = w.of<float>(m * nn), *f2 = w.of<float>(m * nn), *f3 = w.of<float>(m * nn);
        P2 p1 = w.planes(m, n, n, 0), p2 = w.planes(m, n, n, 0), p3 = w.planes(m, n, n, 0);
        QrSpace q;
        qr_space(w, m, n, q);
        float *cd = w.of<float>((long long)m * 4 * tiles * n);
        char *gbase = static_cast<char *>(w.take((size_t)d.grad_plane_bytes));
        most = w.used;
        if (run) {
            if (cudaMemsetAsync(amax, 0, sizeof(float) * 2 * m, s) != cudaSuccess) return record(QT_ERR_LAUNCH);
            QT_TRY(launch_grad_planes(d.grad_stat_items, d.n_grad_stat, d.grad_split_items, d.n_grad_split, d.grads, d.part_amax, d.part_ss, d.gexp,
                                      kTarget, gbase, s));
            // rectified basis: V <- 1.5 V - 0.5 (V V^T) V on its rows
            float *v = f1, *vn = f2;
            P2 pv = p1, pn = p2, pw = p3;
            pv.exp0 = kBasisExp;
            QT_TRY(basis_rows(d, a, m, nullptr, n, v, ld, pv, s, false));
            pw.exp0 = kMaxExp - 4; pw.tmax = kMaxExp;         // entries of V V^T: at most 16
            for (int it = 0; it < d.rect_t1; ++it) {
                Out ow; ow.P = &pw; ow.sym = 1;
                QT_TRY(product(pv, false, pv, true, n, n, n, m, ow, s));
                pn.exp0 = kMaxExp - 3; pn.tmax = kMaxExp; pn.exp = nullptr;   // entries of the result: at most 8
                Out o; o.D = vn; o.C = v; o.ldd = ld; o.strideD = nn; o.P = &pn; o.alpha = -0.5f; o.beta = 1.5f;
                QT_TRY(product(pw, false, pv, false, n, n, n, m, o, s));
                float *tf = v; v = vn; vn = tf;
                P2 tp = pv; pv = pn; pn = tp;
            }
            // L <- V_kept^T diag(S) V_kept, then w1 L + w2 G G^T (G^T G)
            if (launch_chained(k_row_weights, m, 256, 0, s, s.chained, S, max_eig, keep, -1.0f, 0.0f, 8.0f, weights, bound) != cudaSuccess) { cudaGetLastError(); return record(QT_ERR_LAUNCH); }
            count_launch(1);
            P2 ra = pw, rb = pw;                              // planes of the kept rows: two halves of one buffer
            ra.ld = rb.ld = up(n, 16); ra.stride = rb.stride = keep * ra.ld;
            ra.exp0 = kLooseExp; ra.exp = nullptr; rb.exp = exps; rb.exp0 = 0; ra.tmax = rb.tmax = kTarget;
            rb.hi += m * ra.stride; rb.lo += m * ra.stride;
            QT_TRY(to_planes(v, ld, nn, keep, n, m, keep_idx, keep, keep, ra, nullptr, nullptr, &rb, weights, bound, s));
            float *L = vn;
            Out ol; ol.D = L; ol.ldd = ld; ol.strideD = nn; ol.sym = 1;
            QT_TRY(product(ra, true, rb, false, n, n, keep, m, ol, s));
            for (int g = 0; g < d.n_groups; ++g) {
                const qt_refresh_group &gr = d.groups[g];
                P2 pg;
                pg.ld = up(gr.cols, 16); pg.stride = (long long)gr.rows * pg.ld; pg.exp = d.gexp + gr.first; pg.exp0 = 0; pg.tmax = kTarget;
                pg.hi = reinterpret_cast<__half *>(gbase + gr.hi_off); pg.lo = reinterpret_cast<__half *>(gbase + gr.lo_off);
                Out o; o.D = L; o.C = L; o.ldd = ld; o.strideD = nn; o.alpha = d.w2; o.beta = d.w1; o.sym = 1; o.amax = amax; o.slot = gr.slots;
                QT_TRY(product(pg, gr.axis == 1, pg, gr.axis == 0, n, n, gr.axis == 0 ? gr.cols : gr.rows, gr.count, o, s));
            }
            P2 pl = pn;
            pl.exp = exps + m; pl.exp0 = 0; pl.tmax = kTarget;
            QT_TRY(to_planes(L, ld, nn, n, n, m, nullptr, 0, 0, pl, nullptr, amax, nullptr, nullptr, nullptr, s));
            // X = L V^T, its orthonormal basis Q, quotients diag(Q^T L Q)
            float *X = f3;
            Out ox; ox.D = X; ox.ldd = ld; ox.strideD = nn; ox.amax = amax + m;
            QT_TRY(product(pl, false, pv, true, n, n, n, m, ox, s));
            P2 px = pw;
            px.exp = exps + 2 * m; px.exp0 = 0; px.tmax = kTarget;
            QT_TRY(to_planes(X, ld, nn, n, n, m, nullptr, 0, 0, px, nullptr, amax + m, nullptr, nullptr, nullptr, s));
            float *Q = v;
            P2 pq = pv;
            pq.exp = nullptr; pq.exp0 = kBasisExp; pq.tmax = kTarget;
            QT_TRY(qr_batch(m, n, X, px, Q, pq, q, s));
            Out oc; oc.C = Q; oc.ldd = ld; oc.strideD = nn; oc.beta = 1.0f; oc.cd = cd;
            QT_TRY(product(pl, false, pq, false, n, n, n, m, oc, s));
            int size = 2;
            while (size < n) size <<= 1;
            if (launch_chained(k_spectrum, m, 1024, sizeof(unsigned long long) * size, s, s.chained, cd, 4 * tiles, n, keep, S, keep_idx, max_eig) != cudaSuccess) { cudaGetLastError(); return record(QT_ERR_LAUNCH); }
            count_launch(1);
            if (d.bits == 4 && d.blocksize == 64 && n % 16 == 0 && d.stride_codes % 8 == 0) {
                long long ctas = (long long)nb * nb;
                const long long cap = ((long long)device_sm_count() * 6 + m - 1) / m;      // every CTA builds the code tables
                if (ctas > cap) ctas = cap;
                if (launch_chained(k_quantize_transposed, dim3((unsigned)ctas, m), 256, 0, s, s.chained, Q, ld, nn, d.code, n, nb, absmax, (long long)n * nb, codes,
                                   d.stride_codes) != cudaSuccess) { cudaGetLastError(); return record(QT_ERR_LAUNCH); }
                count_launch(1);
            } else {
                if (launch_chained(k_transpose, dim3((n + 31) / 32, (n + 31) / 32, m), 256, 0, s, s.chained, Q, ld, X, n) != cudaSuccess) { cudaGetLastError(); return record(QT_ERR_LAUNCH); }
                count_launch(1);
                QuantArgs qa{X, QT_F32, (long long)n * n, d.code, n, m, d.blocksize, d.bits, absmax, (long long)n * nb, nullptr, 0, codes, d.stride_codes};
                QT_TRY(launch_quantize(qa, s));
            }
            QT_TRY(check_launch());
        }
    }
    if (d.do_root) {
        w.used = mark;
        const long long kn = keep * ld;
        float *f1 = w.of<float>(m * kn), *f2 = w.of<float>(m * kn);
        P2 p1 = w.planes(m, keep, n, 0), p2 = w.planes(m, keep, n, 0), pw = w.planes(m, keep, keep, kMaxExp - 4);
        pw.tmax = kMaxExp;
        const bool fused = d.bits == 4 && d.blocksize == 64 && n % 16 == 0;
        float *P = fused ? nullptr : w.of<float>((long long)m * n * n);
        if (w.used > most) most = w.used;
        if (run) {
            float *r = f1, *rn = f2;
            P2 pr = p1, pn = p2;
            pr.exp0 = kBasisExp;
            QT_TRY(basis_rows(d, a, m, keep_idx, keep, r, ld, pr, s, !d.do_stat));
            for (int it = 0; it < d.rect_t2; ++it) {
                Out ow; ow.P = &pw; ow.sym = 1;
                QT_TRY(product(pr, false, pr, true, keep, keep, n, m, ow, s));
                pn.exp0 = kMaxExp - 3; pn.tmax = kMaxExp;
                Out o; o.D = rn; o.C = r; o.ldd = ld; o.strideD = kn; o.P = &pn; o.alpha = -0.5f; o.beta = 1.5f;
                QT_TRY(product(pw, false, pr, false, keep, n, keep, m, o, s));
                float *tf = r; r = rn; rn = tf;
                P2 tp = pr; pr = pn; pn = tp;
            }
            if (launch_chained(k_row_weights, m, 256, 0, s, s.chained, S, max_eig, keep, d.eps, d.inv_p, 8.0f, weights, bound) != cudaSuccess) { cudaGetLastError(); return record(QT_ERR_LAUNCH); }
            count_launch(1);
            P2 ps = pn;
            ps.exp = exps; ps.exp0 = 0; ps.tmax = kTarget;
            QT_TRY(to_planes(r, ld, kn, keep, n, m, nullptr, 0, keep, ps, weights, bound, nullptr, nullptr, nullptr, s));
            unsigned char *pc = d.prec_codes + (long long)a * d.stride_codes;
            float *pa = d.prec_absmax + (long long)a * n * nb, *pd = d.prec_diag + (long long)a * n;
            if (fused) {
                GemmArgs ga{pr.hi, pr.lo, pr.ld, pr.stride, 1, ps.hi, ps.lo, ps.ld, ps.stride, 1, n, n, keep, m, 1.0f, 0.0f,
                            nullptr, 0, 0, nullptr, 0, 0, nullptr, nullptr, 0, 0};
                GemmExtras x;
                x.f16 = 1; x.kc = 2; x.a_exp = pr.exp; x.b_exp = ps.exp; x.ab_exp0 = pr.exp0 + ps.exp0;
                QuantStateArgs qs{d.code, nullptr, nullptr, nullptr, pc, pa, pd, d.stride_codes, (long long)n * nb, n};
                QT_TRY(launch_gemm_planes(ga, nullptr, nullptr, s, &qs, &x));
            } else {
                Out o; o.D = P; o.ldd = n; o.strideD = (long long)n * n; o.sym = 1;
                QT_TRY(product(pr, true, ps, false, n, n, keep, m, o, s));
                QuantArgs qa{P, QT_F32, (long long)n * n, d.code, n, m, d.blocksize, d.bits, pa, (long long)n * nb, pd, n, pc, d.stride_codes};
                QT_TRY(launch_quantize(qa, s));
            }
        }
    }
    w.used = most;
    return QT_OK;
}

int read_refresh_error(bool clear) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof(int)) != cudaSuccess) return QT_ERR_LAUNCH;
    if (clear && v != 0) {
        int z = 0;
        cudaMemcpyToSymbol(g_gemm_error, &z, sizeof(int));
    }
    return v;
}

static bool refresh_ok(const qt_refresh_desc *d) {
    return d && d->n >= 64 && d->n <= 1216 && d->count > 0 && d->keep > 0 && d->keep <= d->n && (d->bits == 4 || d->bits == 8) &&
           valid_blocksize(d->blocksize) && d->stride_codes % 16 == 0 && d->n_groups >= 0;
}

}  // namespace qt

using namespace qt;

extern "C" {

unsigned long long qt_refresh_workspace_bytes(const qt_refresh_desc *d) {
    if (!refresh_ok(d)) return 0;
    Bump w{nullptr, 0, 0};
    if (refresh_pass(*d, 0, d->count, w, false, nullptr) != QT_OK) return 0;
    return w.used + 256;
}

int qt_refresh_class(const qt_refresh_desc *d, void *workspace, unsigned long long workspace_bytes, void *stream) {
    if (!refresh_ok(d)) return record(QT_ERR_UNSUPPORTED);
    if (!d->stat_codes || !d->stat_absmax || !d->S || !d->keep_idx || !d->max_eig || !d->code || !workspace) return record(QT_ERR_ARG);
    if (d->do_root && (!d->prec_codes || !d->prec_absmax || !d->prec_diag)) return record(QT_ERR_ARG);
    if (workspace_bytes < qt_refresh_workspace_bytes(d)) return record(QT_ERR_ARG);
    Bump w{static_cast<char *>(workspace), 0, (size_t)workspace_bytes};
    return record(refresh_pass(*d, 0, d->count, w, true, static_cast<cudaStream_t>(stream)));
}

}  // extern "C"
