// The part of an optimizer step that runs every time: preconditioned directions P0 G P1 of all gradient blocks, norm
// grafting and the AdamW / SGD tail (reference project paths optimizers/shampoo2.py:234-272, :441-466), in five launches
// whatever the number of parameters and shapes:
//   1 k_apply_stats   largest magnitude of every gradient block and sum of squares of every gradient, in pieces;
//                     largest magnitude of every 4/8-bit preconditioner from its block scales and diagonal;
//   2 k_apply_planes  gradients and preconditioners as scaled fp16 operand planes;
//   3 k_apply_gemm    T = P0 G for all blocks, written as operand planes;
//   4 k_apply_gemm    R = T P1, written in the shape of the parameters, with the sum of squares of every tile;
//   5 k_apply_tail    grafting factor of the tensor, moments, parameters.
// Blocks with an order below 64 (whose preconditioner is a plain fp32 matrix) are multiplied in fp32 by extra CTAs of
// launches 1 and 2.  A launch walks a table of work items that the caller lays out once (addresses, sizes): an ordinary
// step of a small network is bound by launches and host work, one of a large network by HBM, and per-shape launches
// (ResNet-34: 24 shapes, 700 launches with their copies, concatenations and norms) served neither.
#include "quant_device.cuh"
#include "tc_device.cuh"
#include <cuda_fp16.h>
#include <cstring>

namespace qt {

static constexpr int kApplyThreads = 256;

// One work item (80 bytes; mirrored by optimizers/_apply.py).
struct ApplyItem {
    int type, param, rows, cols, ld, aux0, aux1, aux2;
    long long off, p0, p1, p2, p3, p4;
};
enum { kGradStat = 0, kStateExp = 1, kSimtFirst = 2, kSplit = 3, kDequant = 4, kSimtSecond = 5 };

__device__ __forceinline__ float block_sum(float v, float *red) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.0f;
#pragma unroll
    for (int i = 0; i < kApplyThreads / 32; ++i) v += red[i];
    __syncthreads();
    return v;
}
__device__ __forceinline__ float block_max(float v, float *red) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
#pragma unroll
    for (int i = 1; i < kApplyThreads / 32; ++i) v = fmaxf(v, red[i]);
    __syncthreads();
    return v;
}

// Element (r, c) of a stored matrix of order n: bits 32 = plain fp32, else codes with block scales and fp32 diagonal.
__device__ __forceinline__ float state_value(long long var, long long absmax, long long diag, const float *code, int bits, int bs_shift,
                                             int n, int r, int c) {
    const long long e = (long long)r * n + c;
    if (bits == 32) return __ldg(reinterpret_cast<const float *>(var) + e);
    if (diag != 0 && r == c) return __ldg(reinterpret_cast<const float *>(diag) + r);
    const unsigned char *q = reinterpret_cast<const unsigned char *>(var);
    const int nb = (n + (1 << bs_shift) - 1) >> bs_shift;
    const float am = __ldg(reinterpret_cast<const float *>(absmax) + (long long)r * nb + (c >> bs_shift));
    int k;
    if (bits == 8) k = __ldg(q + e);
    else { const int byte = __ldg(q + (e >> 1)); k = (e & 1) ? (byte & 15) : (byte >> 4); }
    return fmaf(__ldg(code + k), am, am == 0.0f ? 0.0f : -0.0f);
}

// One 32 x 32 tile of an fp32 product C = A B (A: M x K, B: K x N), 256 threads, four results each.  `a` and `b` give the
// elements.  The next chunk of 32 k is fetched while this one is multiplied.  Returns the thread's sum of squares.
template <class FA, class FB>
__device__ __forceinline__ float simt_tile(int M, int N, int K, int tm, int tn, FA a, FB b, float *C, long long ldc, float (*As)[33], float (*Bs)[33]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int lc = threadIdx.x & 31, lr = threadIdx.x >> 5;  // chunk elements (lr + 8 q, lc)
    const int m0 = tm * 32, n0 = tn * 32;
    float ra[4], rb[4], acc[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
    auto fetch = [&](int k0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = lr + 8 * q;
            ra[q] = (m0 + r < M && k0 + lc < K) ? a(m0 + r, k0 + lc) : 0.0f;
            rb[q] = (k0 + r < K && n0 + lc < N) ? b(k0 + r, n0 + lc) : 0.0f;
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < K; k0 += 32) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) { As[lr + 8 * q][lc] = ra[q]; Bs[lr + 8 * q][lc] = rb[q]; }
        __syncthreads();
        if (k0 + 32 < K) fetch(k0 + 32);
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            const float a0 = As[ty][k], a1 = As[ty + 16][k], b0 = Bs[k][tx], b1 = Bs[k][tx + 16];
            acc[0][0] = fmaf(a0, b0, acc[0][0]); acc[0][1] = fmaf(a0, b1, acc[0][1]);
            acc[1][0] = fmaf(a1, b0, acc[1][0]); acc[1][1] = fmaf(a1, b1, acc[1][1]);
        }
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int r = m0 + ty + 16 * i, c = n0 + tx + 16 * j;
            if (r < M && c < N) { C[(long long)r * ldc + c] = acc[i][j]; ss = fmaf(acc[i][j], acc[i][j], ss); }
        }
    return ss;
}

// ---- launch 1 ---------------------------------------------------------------------------------
// Gradients are read once here (55 us for the 353 MB of ViT-B/32 at the copy rate); the magnitude has to be known
// before the planes can be scaled, and the same pass yields the norms for the grafting.
__global__ void __launch_bounds__(kApplyThreads)
k_apply_stats(const ApplyItem *__restrict__ items, const long long *__restrict__ grads, const float *__restrict__ code,
              float *__restrict__ part_amax, float *__restrict__ part_ss, int *__restrict__ pexp, int target) {
    __shared__ float red[kApplyThreads / 32];
    __shared__ float As[32][33], Bs[32][33];
    const ApplyItem &it = items[blockIdx.x];
    if (it.type == kGradStat) {
        const float *g = reinterpret_cast<const float *>(grads[it.param]) + it.off;
        float am = 0.0f, s0 = 0.0f, s1 = 0.0f;
        const int rows = it.rows, cols = it.cols, ld = it.ld;
        if ((reinterpret_cast<uintptr_t>(g) & 15) == 0 && (rows == 1 || ld % 4 == 0)) {
            const int c4 = cols / 4, total = rows * c4;
#pragma unroll 4
            for (int t = threadIdx.x; t < total; t += kApplyThreads) {
                const int r = rows == 1 ? 0 : t / c4;
                const float4 x = __ldg(reinterpret_cast<const float4 *>(g + (long long)r * ld + 4 * (t - r * c4)));
                am = fmaxf(am, fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))));
                s0 = fmaf(x.x, x.x, fmaf(x.y, x.y, s0));
                s1 = fmaf(x.z, x.z, fmaf(x.w, x.w, s1));
            }
            const int tail = cols & 3;
            for (int t = threadIdx.x; t < rows * tail; t += kApplyThreads) {
                const float x = g[(long long)(t / tail) * ld + 4 * c4 + t % tail];
                am = fmaxf(am, fabsf(x));
                s0 = fmaf(x, x, s0);
            }
        } else {
            const int total = rows * cols;
#pragma unroll 4
            for (int t = threadIdx.x; t < total; t += kApplyThreads) {
                const int r = t / cols;
                const float x = __ldg(g + (long long)r * ld + (t - r * cols));
                am = fmaxf(am, fabsf(x));
                s0 = fmaf(x, x, s0);
            }
        }
        am = block_max(am, red);
        const float ss = block_sum(s0 + s1, red);
        if (threadIdx.x == 0) { part_amax[it.aux0] = am; part_ss[it.aux0] = ss; }
    } else if (it.type == kStateExp) {
        const float *am = reinterpret_cast<const float *>(it.p0), *dg = reinterpret_cast<const float *>(it.p1);
        float v = 0.0f;
#pragma unroll 4
        for (int t = threadIdx.x; t < it.rows; t += kApplyThreads) v = fmaxf(v, fabsf(__ldg(am + t)));
        if (dg)
#pragma unroll 2
            for (int t = threadIdx.x; t < it.cols; t += kApplyThreads) v = fmaxf(v, fabsf(__ldg(dg + t)));
        v = block_max(v, red);
        if (threadIdx.x == 0) pexp[it.aux0] = exponent_for(v, target);
    } else {                                                  // T = P0 G in fp32
        const float *g = reinterpret_cast<const float *>(grads[it.param]) + it.off;
        const int bits = it.aux0 & 255, shift = it.aux0 >> 8, m = it.rows, ld = it.ld;
        simt_tile(m, it.cols, m, it.aux1, it.aux2,
                  [&](int r, int c) { return state_value(it.p0, it.p1, it.p2, code, bits, shift, m, r, c); },
                  [&](int r, int c) { return __ldg(g + (long long)r * ld + c); },
                  reinterpret_cast<float *>(it.p4), it.cols, As, Bs);
    }
}

// ---- launch 2 ---------------------------------------------------------------------------------
__device__ __forceinline__ void store_f16_pair(__half *hi, __half *lo, const float (&v)[16]) {
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

// Rows of planes are padded to 16 elements, so every thread writes 16 columns with one 256-bit store per plane whatever
// the order.  The codes of an order that is no multiple of 16 start at any nibble of a word: three aligned words and
// two funnel shifts give the sixteen codes.
__global__ void __launch_bounds__(kApplyThreads)
k_apply_planes(const ApplyItem *__restrict__ items, const long long *__restrict__ grads, const float *__restrict__ code,
               const float *__restrict__ part_amax, float *__restrict__ part_ss, const int *__restrict__ pexp, int *__restrict__ gexp, int target,
               long long plane_base) {
    __shared__ float red[kApplyThreads / 32];
    __shared__ __align__(16) unsigned char raw[2 * 32 * 33 * 4];
    float2 *pair_lut = reinterpret_cast<float2 *>(raw);
    const ApplyItem &it = items[blockIdx.x];
    if (it.type == kSplit) {
        float am = 0.0f;
        for (int t = threadIdx.x; t < it.aux1; t += kApplyThreads) am = fmaxf(am, __ldg(part_amax + it.aux0 + t));
        am = block_max(am, red);
        const int e = exponent_for(am, target);
        if (it.p3 && threadIdx.x == 0) gexp[it.aux2] = e;     // the block's first item
        const float two_e = exp2f((float)e);
        const float *g = reinterpret_cast<const float *>(grads[it.param]) + it.off;
        __half *hi = reinterpret_cast<__half *>(plane_base + it.p0), *lo = reinterpret_cast<__half *>(plane_base + it.p1);
        const int rows = it.rows, cols = it.cols, ld = it.ld;
        const long long ldp = it.p2;
        const bool vec = (reinterpret_cast<uintptr_t>(g) & 31) == 0 && ld % 8 == 0;
        const int c16 = (cols + 15) >> 4, total = rows * c16;
        float worst = 0.0f;
#pragma unroll 2
        for (int t = threadIdx.x; t < total; t += kApplyThreads) {
            const int r = t / c16, c = (t - r * c16) * 16;
            const float *src = g + (long long)r * ld + c;
            float v[16];
            if (vec && c + 16 <= cols) { ldg256f(src, v); ldg256f(src + 8, v + 8); }
            else {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = c + j < cols ? __ldg(src + j) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                v[j] = fminf(fmaxf(v[j] * two_e, -65000.0f), 65000.0f);
                worst = fmaxf(worst, fabsf(v[j]));
            }
            store_f16_pair(hi + r * ldp + c, lo + r * ldp + c, v);
        }
        if (worst >= 65000.0f) atomicCAS(&g_gemm_error, 0, QT_ERR_RANGE);
    } else if (it.type == kDequant) {
        const int bits = it.aux0 & 255, shift = it.aux0 >> 8, n = it.cols;
        float *code_s = reinterpret_cast<float *>(raw);
        if (bits == 4) { const int i = threadIdx.x; pair_lut[i] = make_float2(__ldg(code + (i >> 4)), __ldg(code + (i & 15))); }
        else code_s[threadIdx.x] = __ldg(code + threadIdx.x);
        __syncthreads();
        const float two_e = exp2f((float)__ldg(pexp + it.aux1));
        const unsigned char *in = reinterpret_cast<const unsigned char *>(it.p0);
        const float *absmax = reinterpret_cast<const float *>(it.p1), *diag = reinterpret_cast<const float *>(it.p2);
        __half *hi = reinterpret_cast<__half *>(it.p3), *lo = reinterpret_cast<__half *>(it.p4);
        const int row0 = (int)it.off, rows = it.rows, nb = (n + (1 << shift) - 1) >> shift;
        const long long ldp = it.ld;
        const int c16 = (n + 15) >> 4, total = rows * c16;
        const bool even = n % 16 == 0;
        const unsigned last_word = ((unsigned)n * (unsigned)n - 1u) >> 3;
#pragma unroll 2
        for (int t = threadIdx.x; t < total; t += kApplyThreads) {
            const int rr = t / c16, r = row0 + rr, c = (t - rr * c16) * 16;
            const unsigned f = (unsigned)r * (unsigned)n + (unsigned)c;     // below 2^31
            const float am = __ldg(absmax + (long long)r * nb + (c >> shift));
            const float z = (am == 0.0f) ? 0.0f : -0.0f;      // exact +0.0 for all-zero blocks
            float v[16];
            if (bits == 4) {
                unsigned w0, w1;                              // sixteen codes, the first in the top nibble
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
            if (diag && (unsigned)(r - c) < 16u) {
                const float d = __ldg(diag + r);
#pragma unroll
                for (int j = 0; j < 16; ++j) if (c + j == r) v[j] = d;
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] *= two_e;
            store_f16_pair(hi + r * ldp + c, lo + r * ldp + c, v);
        }
    } else {                                                  // R = T P1 in fp32
        float (*As)[33] = reinterpret_cast<float (*)[33]>(raw);
        float (*Bs)[33] = reinterpret_cast<float (*)[33]>(raw + 32 * 33 * 4);
        const float *T = reinterpret_cast<const float *>(it.p4);
        const int bits = it.aux0 & 255, shift = it.aux0 >> 8, k = it.cols;
        const float ss = simt_tile(it.rows, k, k, it.aux1, it.aux2,
                                   [&](int r, int c) { return __ldg(T + (long long)r * k + c); },
                                   [&](int r, int c) { return state_value(it.p0, it.p1, it.p2, code, bits, shift, k, r, c); },
                                   reinterpret_cast<float *>(it.p3), it.ld, As, Bs);
        const float sum = block_sum(ss, red);
        if (threadIdx.x == 0) part_ss[it.off] = sum;
    }
}

// ---- launches 3 and 4 ---------------------------------------------------------------------------
// Products of all block shapes of the step in one persistent grid: C = A B with A row-major (k contiguous), B row-major
// (n contiguous), both scaled fp16 pairs; three MMAs per k-slice, accumulation chains of 128 k added up in registers,
// as in k_gemm_bf16x3.  A group holds the blocks of one shape; its operand maps lie in device memory.
struct alignas(128) ApplyGroup {
    CUtensorMap a[2], b[2];
    int M, N, K, batch, tiles_m, tiles_n, tile0, rel;         // tile0: first tile of the group; rel: exponent of plane results
    const int *a_exp, *b_exp;                                 // per block
    __half *Phi, *Plo; long long ldp, strideP; int *out_exp;   // result as planes (T), or
    float *const *D; long long ldd; float *part; int wide, pad; // in place (R, one address per block), with the sums of squares
};

template <int BN> struct ApplyCfg {
    static constexpr int BM = 128, BK = 64, KC = 2;
    static constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
    static constexpr int STAGE = 2 * (A_BYTES + B_BYTES), STAGES = 12 * A_BYTES / STAGE;
    static constexpr int EC = BN / 2, EPI = 8, NACC = 512 / BN;
    // 128 partial sums a thread need more than the 168 registers that ten warps get: two idle warps complete the producers'
    // warpgroup, which hands registers to the epilogue (launch: 384 x 168 = 256 x 224 + 128 x 56)
    static constexpr bool REGS = BN == 256;
    static constexpr int THREADS = (EPI + (REGS ? 4 : 2)) * 32;
    static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
};
static constexpr int kMaxGroups = 256;

template <int BN>
__global__ void __launch_bounds__(ApplyCfg<BN>::THREADS, 1)
k_apply_gemm(const ApplyGroup *__restrict__ groups, const int *__restrict__ tile_start, int ngroups) {
    using Cfg = ApplyCfg<BN>;
    constexpr int STAGES = Cfg::STAGES, EPI = Cfg::EPI, NACC = Cfg::NACC, EC = Cfg::EC, KC = Cfg::KC, BM = Cfg::BM, BK = Cfg::BK;
    __shared__ int starts[kMaxGroups + 1];
    extern __shared__ unsigned char smem_raw[];
    const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *aligned = smem_raw + (base - smem_u32(smem_raw));
    unsigned long long *bars = reinterpret_cast<unsigned long long *>(aligned + STAGES * Cfg::STAGE);
    unsigned *tmem_slot = reinterpret_cast<unsigned *>(bars + 2 * STAGES + 2 * NACC);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const unsigned bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (STAGES + s); };
    auto acc_full = [&](int a) { return bar0 + 8u * (2 * STAGES + a); };
    auto acc_empty = [&](int a) { return bar0 + 8u * (2 * STAGES + NACC + a); };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // an earlier wait expired: drain fast (all threads or none, the epilogue waits for registers)
    if (__syncthreads_or(*reinterpret_cast<volatile int *>(&g_gemm_error) == QT_ERR_TIMEOUT)) return;
    for (int i = threadIdx.x; i <= ngroups; i += Cfg::THREADS) starts[i] = tile_start[i];
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int a = 0; a < NACC; ++a) { mbar_init(acc_full(a), 1); mbar_init(acc_empty(a), EPI); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == EPI + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_base = *tmem_slot;
    const int num_tiles = starts[ngroups];

    if (warp >= EPI) {
    if constexpr (Cfg::REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == EPI) {
        if (lane == 0) {                                      // TMA producer
            unsigned it = 0;
            bool ok = true;
            int gi = 0;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                while (tile >= starts[gi + 1]) ++gi;
                const ApplyGroup &g = groups[gi];
                int tm, tn, b;
                tile_coords(tile - starts[gi], g.tiles_m, g.tiles_n, tm, tn, b);
                const int m0 = tm * BM, n0 = tn * BN, num_kb = (g.K + BK - 1) / BK, ncols = g.N - n0;
                const int bchunks = ncols >= BN ? BN / 64 : (ncols + 63) / 64;       // 64-column pieces of B that exist
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    ok = mbar_wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, abort_flag);
                    if (!ok) break;
                    const unsigned stage = base + s * Cfg::STAGE;
                    mbar_expect_tx(full_bar(s), 2 * (Cfg::A_BYTES + bchunks * (64 * BK * 2)));
#pragma unroll
                    for (int pl = 0; pl < 2; ++pl) {
                        tma_load_3d(stage + pl * Cfg::A_BYTES, &g.a[pl], full_bar(s), kb * BK, m0, b);
                        const unsigned tb = stage + 2 * Cfg::A_BYTES + pl * Cfg::B_BYTES;
                        for (int c = 0; c < bchunks; ++c) tma_load_3d(tb + c * (64 * BK * 2), &g.b[pl], full_bar(s), n0 + 64 * c, kb * BK, b);
                    }
                }
            }
        }
    } else if (warp == EPI + 1) {
        if (lane == 0) {                                      // MMA issuer
            // fp32 accumulation, fp16 operands, A K-major, B MN-major
            const unsigned idesc0 = (1u << 4) | (1u << 16) | ((unsigned)(BM >> 4) << 24);
            unsigned long long dA[2], dB[2];
#pragma unroll
            for (int pl = 0; pl < 2; ++pl) {
                dA[pl] = smem_desc(base + pl * Cfg::A_BYTES, 16u, 1024u);
                dB[pl] = smem_desc(base + 2 * Cfg::A_BYTES + pl * Cfg::B_BYTES, 8192u, 1024u);
            }
            unsigned it = 0;
            bool ok = true;
            int j = 0, gi = 0;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                while (tile >= starts[gi + 1]) ++gi;
                const ApplyGroup &g = groups[gi];
                int tm, tn, b;
                tile_coords(tile - starts[gi], g.tiles_m, g.tiles_n, tm, tn, b);
                const int num_kb = (g.K + BK - 1) / BK;
                const int ncur = min(BN, (g.N - tn * BN + 15) & ~15);    // a ragged last band multiplies its own columns only
                const unsigned idesc = idesc0 | ((unsigned)(ncur >> 3) << 17);
                for (int kb = 0; kb < num_kb && ok; ++j) {
                    const int acc = j % NACC;
                    ok = mbar_wait(acc_empty(acc), ((j / NACC) & 1) ^ 1, abort_flag);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned tmem_acc = tmem_base + (unsigned)(acc * BN);
                    const int kend = min(num_kb, kb + KC);
                    for (bool fresh = true; kb < kend; ++kb, ++it, fresh = false) {
                        const int s = it % STAGES;
                        ok = mbar_wait(full_bar(s), (it / STAGES) & 1, abort_flag);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const unsigned long long soff = (unsigned long long)((unsigned)(s * Cfg::STAGE) >> 4);
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k) {
                            const unsigned long long ao = soff + k * 2u, bo = soff + k * 128u;
                            umma_bf16(tmem_acc, dA[0] + ao, dB[1] + bo, idesc, fresh && k == 0 ? 0u : 1u);
                            umma_bf16(tmem_acc, dA[1] + ao, dB[0] + bo, idesc, 1u);
                            umma_bf16(tmem_acc, dA[0] + ao, dB[0] + bo, idesc, 1u);
                        }
                        umma_commit(empty_bar(s));
                    }
                    if (ok) umma_commit(acc_full(acc));
                }
            }
        }
    }
    } else {                                                  // epilogue: warp e holds rows 32 (e & 3) .., columns EC (e >> 2) ..
        if constexpr (Cfg::REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        const int quad = warp & 3, seg = warp >> 2;
        int j = 0, gi = 0;
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
            while (tile >= starts[gi + 1]) ++gi;
            const ApplyGroup &g = groups[gi];
            int tm, tn, b;
            tile_coords(tile - starts[gi], g.tiles_m, g.tiles_n, tm, tn, b);
            const int row = tm * BM + quad * 32 + lane, n0 = tn * BN + seg * EC;
            const int valid = min(EC, g.N - n0), nchunks = ((g.K + BK - 1) / BK + KC - 1) / KC;
            float sum[EC];
#pragma unroll
            for (int q = 0; q < EC; ++q) sum[q] = 0.0f;
            bool ok = true;
            for (int ch = 0; ch < nchunks; ++ch, ++j) {
                const int acc = j % NACC;
                ok = mbar_wait_warp(acc_full(acc), (j / NACC) & 1, abort_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned tmem_acc = tmem_base + (unsigned)(acc * BN + seg * EC) + ((unsigned)(quad * 32) << 16);
#pragma unroll
                for (int c = 0; c < EC / 32; ++c) {
                    if (c * 32 < valid) {
                        float v[32];
                        tmem_ld32(tmem_acc + (unsigned)(c * 32), v);
#pragma unroll
                        for (int q = 0; q < 32; ++q) sum[c * 32 + q] += v[q];
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty(acc)) : "memory");
            }
            if (!ok) break;
            const int e_in = __ldg(g.a_exp + b) + __ldg(g.b_exp + b);
            float ss = 0.0f;
            if (g.Phi) {
                if (tm == 0 && tn == 0 && warp == 0 && lane == 0) g.out_exp[b] = e_in + g.rel;
                if (row < g.M) {
                    // entry = value * 2^(e_in + rel) and the accumulator holds value * 2^e_in: one exact factor
                    const float f = exp2f((float)g.rel);
                    const long long o = (long long)b * g.strideP + (long long)row * g.ldp + n0;
#pragma unroll
                    for (int q = 0; q < EC; q += 16) {
                        if (q < valid) {                      // rows of planes are padded to 16 columns
                            float v[16];
#pragma unroll
                            for (int t = 0; t < 16; ++t) v[t] = sum[q + t] * f;
                            unsigned H[8], L[8];
#pragma unroll
                            for (int t = 0; t < 8; ++t) {
                                const __half h0 = __float2half_rn(v[2 * t]), h1 = __float2half_rn(v[2 * t + 1]);
                                const __half l0 = __float2half_rn(v[2 * t] - __half2float(h0)), l1 = __float2half_rn(v[2 * t + 1] - __half2float(h1));
                                H[t] = (unsigned)__half_as_ushort(h0) | ((unsigned)__half_as_ushort(h1) << 16);
                                L[t] = (unsigned)__half_as_ushort(l0) | ((unsigned)__half_as_ushort(l1) << 16);
                            }
                            stg256u(reinterpret_cast<unsigned *>(g.Phi + o + q), H);
                            stg256u(reinterpret_cast<unsigned *>(g.Plo + o + q), L);
                        }
                    }
                }
            } else {
                if (row < g.M) {
                    const float f = exp2f((float)-e_in);
                    float *d = g.D[b] + (long long)row * g.ldd + n0;
#pragma unroll
                    for (int q = 0; q < EC; q += 16) {
                        if (q < valid) {
                            float o[16];
#pragma unroll
                            for (int t = 0; t < 16; ++t) {
                                o[t] = sum[q + t] * f;
                                if (q + t < valid) ss = fmaf(o[t], o[t], ss);
                            }
                            if (g.wide && q + 16 <= valid) { stg256f(d + q, o); stg256f(d + q + 8, o + 8); }
                            else {
#pragma unroll
                                for (int t = 0; t < 16; ++t) if (q + t < valid) d[q + t] = o[t];
                            }
                        }
                    }
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
                if (lane == 0) g.part[(long long)(tile - starts[gi]) * EPI + warp] = ss;
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    if (warp == EPI + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// ---- launch 5 ---------------------------------------------------------------------------------
// One entry per parameter (80 bytes; mirrored by optimizers/_apply.py).
struct ApplyTensor {
    long long p, m, v, d;                                     // d == 0: the direction is the gradient itself
    long long numel;
    int param, flags;                                         // flags: 1 = grafted, 2 = the decayed direction is written back to the gradient
    int g0, g1;                                               // pieces of the gradient's sum of squares
    int r0, r1;                                               // ranges (first, count) of pieces of the direction's sum of squares
    long long pad;
};
struct ApplyTailParams {
    const ApplyTensor *tensors; const int *chunk_tensor, *chunk_index; const int2 *ranges; const float *part; const long long *grads;
    int chunk_elems, kind, nesterov;                          // kind: 0 AdamW, 1 SGD
    const float *scalars;                                     // AdamW factors in device memory (graph replay), or null: s0, s1, s2
    float s0, s1, s2, beta1, beta2, a1, a2, eps, lr, momentum, weight_decay;
};

// The grafting factor ||G|| / (||R|| + 1e-12) is formed by every CTA from the tensor's pieces (a few hundred floats,
// read beside the first data) instead of by a launch of its own: 28 bytes per element of AdamW traffic are the bound.
template <int KIND>
__global__ void __launch_bounds__(kApplyThreads)
k_apply_tail(const ApplyTailParams q) {
    __shared__ float red[kApplyThreads / 32];
    const ApplyTensor &t = q.tensors[q.chunk_tensor[blockIdx.x]];
    const long long begin = (long long)q.chunk_index[blockIdx.x] * q.chunk_elems;
    const long long end = min(begin + q.chunk_elems, t.numel);
    float *p = reinterpret_cast<float *>(t.p), *m = reinterpret_cast<float *>(t.m), *v = reinterpret_cast<float *>(t.v);
    float *grad = reinterpret_cast<float *>(q.grads[t.param]);
    const float *d = t.d ? reinterpret_cast<const float *>(t.d) : grad;
    float factor = 1.0f;
    if (t.flags & 1) {
        float gs = 0.0f, ds = 0.0f;
        for (int i = t.g0 + threadIdx.x; i < t.g1; i += kApplyThreads) gs += __ldg(q.part + i);
        for (int r = t.r0; r < t.r1; ++r) {
            const int2 range = __ldg(q.ranges + r);
            for (int i = threadIdx.x; i < range.y; i += kApplyThreads) ds += __ldg(q.part + range.x + i);
        }
        gs = block_sum(gs, red);
        ds = t.r1 > t.r0 ? block_sum(ds, red) : gs;
        factor = sqrtf(gs) / (sqrtf(ds) + 1e-12f);
    }
    const float c0 = q.scalars ? q.scalars[0] : q.s0, c1 = q.scalars ? q.scalars[1] : q.s1, c2 = q.scalars ? q.scalars[2] : q.s2;
    auto update = [&](float &pp, float &dd, float &mm, float &vv) {
        dd *= factor;
        if constexpr (KIND == 0) {
            const float p1 = pp * c2;
            mm = fmaf(q.a1, dd, mm * q.beta1);
            vv = fmaf(q.a2 * dd, dd, vv * q.beta2);
            const float denom = sqrtf(vv) * c0 + q.eps;
            pp = fmaf(c1, mm / denom, p1);
        } else {
            if (q.weight_decay != 0.0f) dd = fmaf(q.weight_decay, pp, dd);
            mm = fmaf(mm, q.momentum, dd);
            pp = fmaf(-q.lr, q.nesterov ? fmaf(q.momentum, mm, dd) : mm, pp);
        }
    };
    const bool back = KIND == 1 && (t.flags & 2);
    const bool vec = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(d) | reinterpret_cast<uintptr_t>(m) |
                       reinterpret_cast<uintptr_t>(v)) & 15) == 0;       // chunk_elems is a multiple of 4
    long long i = begin + (vec ? 4ll : 1ll) * threadIdx.x;
    if (vec) {
        const long long end4 = begin + ((end - begin) & ~3ll);
#pragma unroll 2
        for (; i < end4; i += 4ll * kApplyThreads) {
            float4 P = *reinterpret_cast<float4 *>(p + i), M = *reinterpret_cast<float4 *>(m + i), V = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if constexpr (KIND == 0) V = *reinterpret_cast<float4 *>(v + i);
            float4 D = *reinterpret_cast<const float4 *>(d + i);
            update(P.x, D.x, M.x, V.x); update(P.y, D.y, M.y, V.y); update(P.z, D.z, M.z, V.z); update(P.w, D.w, M.w, V.w);
            *reinterpret_cast<float4 *>(p + i) = P;
            *reinterpret_cast<float4 *>(m + i) = M;
            if constexpr (KIND == 0) *reinterpret_cast<float4 *>(v + i) = V;
            if (back) *reinterpret_cast<float4 *>(grad + i) = D;
        }
        i = end4 + threadIdx.x;
    }
    for (; i < end; i += kApplyThreads) {
        float P = p[i], M = m[i], V = KIND == 0 ? v[i] : 0.0f, D = d[i];
        update(P, D, M, V);
        p[i] = P;
        m[i] = M;
        if constexpr (KIND == 0) v[i] = V;
        if (back) grad[i] = D;
    }
}

// Gradient blocks as operand planes for the statistics: the pieces' magnitudes, then the planes at plane_base + the
// items' offsets.
int launch_grad_planes(const void *stat_items, int n_stat, const void *split_items, int n_split, const long long *grads, float *part_amax,
                       float *part_ss, int *gexp, int target, void *plane_base, cudaStream_t s) {
    if (n_stat <= 0 || n_split <= 0) return record(QT_OK);
    if (!stat_items || !split_items || !grads || !part_amax || !part_ss || !gexp || !plane_base) return record(QT_ERR_ARG);
    k_apply_stats<<<n_stat, kApplyThreads, 0, s>>>(static_cast<const ApplyItem *>(stat_items), grads, nullptr, part_amax, part_ss, nullptr, target);
    k_apply_planes<<<n_split, kApplyThreads, 0, s>>>(static_cast<const ApplyItem *>(split_items), grads, nullptr, part_amax, part_ss, nullptr, gexp, target,
                                                     reinterpret_cast<long long>(plane_base));
    count_launch(2);
    return check_launch();
}

static bool prepare_apply() {
    static PerDeviceOnce done;
    const int dev = current_device();
    if (done.pending(dev)) {
        if (cudaFuncSetAttribute(k_apply_gemm<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, ApplyCfg<128>::SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(k_apply_gemm<192>, cudaFuncAttributeMaxDynamicSharedMemorySize, ApplyCfg<192>::SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(k_apply_gemm<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, ApplyCfg<256>::SMEM) != cudaSuccess)
            return false;
        done.mark(dev);
    }
    return true;
}

static void launch_apply_gemm(const void *groups, const int *tiles, int ngroups, int ntiles, int bn, cudaStream_t s) {
    const int sms = device_sm_count();
    const unsigned grid = (unsigned)(ntiles < sms ? ntiles : sms);
    if (bn == 256)
        k_apply_gemm<256><<<grid, ApplyCfg<256>::THREADS, ApplyCfg<256>::SMEM, s>>>(static_cast<const ApplyGroup *>(groups), tiles, ngroups);
    else if (bn == 192)
        k_apply_gemm<192><<<grid, ApplyCfg<192>::THREADS, ApplyCfg<192>::SMEM, s>>>(static_cast<const ApplyGroup *>(groups), tiles, ngroups);
    else
        k_apply_gemm<128><<<grid, ApplyCfg<128>::THREADS, ApplyCfg<128>::SMEM, s>>>(static_cast<const ApplyGroup *>(groups), tiles, ngroups);
    count_launch(1);
}

int read_apply_error(bool clear) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof(int)) != cudaSuccess) return QT_ERR_LAUNCH;
    if (clear && v != 0) {
        int z = 0;
        cudaMemcpyToSymbol(g_gemm_error, &z, sizeof(int));
    }
    return v;
}

}  // namespace qt

using namespace qt;

extern "C" {

int qt_apply_group(void *out, const void *Ahi, const void *Alo, long long lda, long long strideA, const void *Bhi, const void *Blo,
                   long long ldb, long long strideB, int M, int N, int K, int batch, int bn, int tile0,
                   const int *a_exp, const int *b_exp, void *Phi, void *Plo, long long ldp, long long strideP, int *out_exp, int rel,
                   void *D, long long ldd, int wide, float *part) {
    static_assert(sizeof(ApplyGroup) == QT_APPLY_GROUP_BYTES && sizeof(ApplyItem) == 80 && sizeof(ApplyTensor) == 72, "table layouts");
    if (!out || !Ahi || !Alo || !Bhi || !Blo || M <= 0 || N <= 0 || K <= 0 || batch <= 0 || (bn != 128 && bn != 192 && bn != 256)) return record(QT_ERR_ARG);
    if (lda % 8 || ldb % 8 || strideA % 8 || strideB % 8 || !a_exp || !b_exp || (!Phi && (!D || !part)) || (Phi && (!Plo || !out_exp || ldp % 16)))
        return record(QT_ERR_ARG);
    ApplyGroup g;
    memset(&g, 0, sizeof(g));
    const void *A[2] = {Ahi, Alo}, *B[2] = {Bhi, Blo};
    for (int i = 0; i < 2; ++i)
        if (!make_map(&g.a[i], A[i], K, M, batch, lda, strideA, 64, 128, true) || !make_map(&g.b[i], B[i], N, K, batch, ldb, strideB, 64, 64, true))
            return record(QT_ERR_LAUNCH);
    g.M = M; g.N = N; g.K = K; g.batch = batch;
    g.tiles_m = (M + 127) / 128; g.tiles_n = (N + bn - 1) / bn; g.tile0 = tile0; g.rel = rel;
    g.a_exp = a_exp; g.b_exp = b_exp;
    g.Phi = static_cast<__half *>(Phi); g.Plo = static_cast<__half *>(Plo); g.ldp = ldp; g.strideP = strideP; g.out_exp = out_exp;
    g.D = static_cast<float *const *>(D); g.ldd = ldd; g.part = part; g.wide = wide;
    memcpy(out, &g, sizeof(g));
    return record(QT_OK);
}

int qt_apply_run(const qt_apply_desc *d, void *stream) {
    if (!d || d->n_stat_items < 0 || d->n_waves < 0 || (d->n_waves > 0 && !d->waves) || !d->grads) return record(QT_ERR_ARG);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (!prepare_apply()) return record(QT_ERR_LAUNCH);
    if (d->n_stat_items > 0) {
        k_apply_stats<<<d->n_stat_items, kApplyThreads, 0, s>>>(static_cast<const ApplyItem *>(d->stat_items), d->grads, d->code, d->part_amax,
                                                               d->part_ss, d->pexp, d->target);
        count_launch(1);
    }
    for (int w = 0; w < d->n_waves; ++w) {
        const qt_apply_wave &v = d->waves[w];
        if (v.n_groups > kMaxGroups) return record(QT_ERR_UNSUPPORTED);
        if (v.n_plane_items > 0) {
            k_apply_planes<<<v.n_plane_items, kApplyThreads, 0, s>>>(static_cast<const ApplyItem *>(v.plane_items), d->grads, d->code, d->part_amax,
                                                                    d->part_ss, d->pexp, d->gexp, d->target, 0);
            count_launch(1);
        }
        if (v.n_groups > 0) {
            launch_apply_gemm(v.groups1, v.tiles1, v.n_groups, v.n_tiles1, v.bn1, s);
            launch_apply_gemm(v.groups2, v.tiles2, v.n_groups, v.n_tiles2, v.bn2, s);
        }
    }
    if (d->n_chunks > 0) {
        ApplyTailParams q;
        q.tensors = static_cast<const ApplyTensor *>(d->tensors); q.chunk_tensor = d->chunk_tensor; q.chunk_index = d->chunk_index;
        q.ranges = static_cast<const int2 *>(d->ranges); q.part = d->part_ss; q.grads = d->grads; q.chunk_elems = d->chunk_elems;
        q.kind = d->kind; q.nesterov = d->nesterov; q.scalars = d->scalars; q.s0 = d->s0; q.s1 = d->s1; q.s2 = d->s2;
        q.beta1 = d->beta1; q.beta2 = d->beta2; q.a1 = d->a1; q.a2 = d->a2; q.eps = d->eps;
        q.lr = d->lr; q.momentum = d->momentum; q.weight_decay = d->weight_decay;
        if (d->kind == 0) k_apply_tail<0><<<d->n_chunks, kApplyThreads, 0, s>>>(q);
        else k_apply_tail<1><<<d->n_chunks, kApplyThreads, 0, s>>>(q);
        count_launch(1);
    }
    return check_launch();
}

}  // extern "C"
