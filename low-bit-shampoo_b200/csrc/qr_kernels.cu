// Batched Householder panel factorisation for the eigenbasis refresh of the statistics.
//
// The reference orthonormalises L V with torch.linalg.qr (reference project path
// qtensor/utils.py:157), i.e. one cuSOLVER geqrf + orgqr per matrix.  Here a whole order
// class is factorised together: this kernel factors one 32-column panel of every matrix
// of the batch (one CTA per matrix, the panel resident in shared memory) and emits the
// Householder vectors V (unit lower trapezoidal, explicit zeros and ones) and the
// triangular factor T of the compact-WY form  H_1 .. H_w = I - V T V^T.  The trailing
// update and the accumulation of Q are batched matrix products issued by the caller.
//
// Conventions are LAPACK's (slarfg / slarft, forward, columnwise): beta = -sign(alpha)
// * ||x||, tau = (beta - alpha) / beta, v = x / (alpha - beta) with v_0 = 1; a column
// that is already zero below the diagonal gets tau = 0.
#include "quant_device.cuh"
#include <cuda_fp16.h>

namespace qt {

// Operand planes of an outer block's Householder vectors, written by the panel kernels beside V itself: scaled fp16
// pairs (entries <= 1, so the exponent is fixed), [matrix][n - J0 rows][pitch ld], the panel's columns at col0.  Rows above
// the panel inside the block are written as zeros.
struct PanelPlanes { __half *hi, *lo; long long ld, stride; int col0, rows_above; float scale; };

__device__ __forceinline__ void store_panel_planes(const PanelPlanes &pp, const float *P, int m, int w, int warps) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (!pp.hi || lane >= w) return;
    __half *hi = pp.hi + (long long)blockIdx.x * pp.stride + pp.col0 + lane, *lo = pp.lo + (long long)blockIdx.x * pp.stride + pp.col0 + lane;
    for (int r = warp; r < m + pp.rows_above; r += warps) {
        const float x = r < pp.rows_above ? 0.0f : P[(r - pp.rows_above) * 33 + lane] * pp.scale;
        const __half h = __float2half_rn(x);
        hi[(long long)r * pp.ld] = h;
        lo[(long long)r * pp.ld] = __float2half_rn(x - __half2float(h));
    }
}

static constexpr int kPanel = 32;
static constexpr int kQrThreads = 1024;                    // one warp per panel column
static constexpr int kMaxRowsPerLane = 38;                 // panel rows <= 32 * 38 = 1216
static int g_panel_blocked = 1;                            // test hook: 0 = the kernel with one column per warp
void set_panel_blocked(int on) { g_panel_blocked = on; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// The kernel with one column per warp, kept as the independent form that tests compare the panel kernel with
// (qt_panel_force_form).  Register-resident panel: warp c owns column c, lane l holds rows l, l+32, ... of it for the
// whole factorisation: the first RPL of them in registers, RS more (tall panels only) in the
// column's slots of the shared staging buffer, so that the register budget of a 1024-thread CTA
// (64 per thread) is never exceeded.  Per column step the pivot warp builds its Householder
// vector and publishes it once through a double-buffered shared-memory vector; the warps to
// its right apply the reflector to their own column, the warps to its left (already final)
// take the dot product v_i . v_c needed for the triangular factor T, and warp 0 fills in
// column c-1 of T meanwhile (slarft recurrence), off the critical path.  One barrier per step;
// every reduction chain is split over four accumulators.
//
// Fused form (prev_w > 0): before anything is factored, the block reflector of the PREVIOUS panel
// of the same outer block (Householder vectors in V's columns j0-prev_w .. j0-1, rows j0-prev_w ..
// n-1; its triangular factor Tprev) is applied to 32-column chunks of the rest of the outer block:
//     C <- (I - Vp Tp^T Vp^T) C,   C = A[j0-prev_w : n, j0 + 32 chunk : ...]
// CTA (matrix, chunk) updates chunk `chunk` (written back to A); chunk 0 is the new panel, which
// its CTA goes on to factor from shared memory.  This replaces the three library products per
// panel that a separate rank-32 update needs, and the CTAs of chunks 1.. fill otherwise idle SMs.
template <int RPL, int RS>
__global__ void __launch_bounds__(kQrThreads, 1)
k_householder_panel(float *__restrict__ Abase, long long strideA, int n, int ld, int j0, int w,
                    float *__restrict__ Vbase, long long strideV, float *__restrict__ Tbase, long long strideT,
                    int prev_w, const float *__restrict__ Tprev_base, int block_end, const PanelPlanes planes) {
    constexpr int RT = RPL + RS;
    extern __shared__ float sm[];
    const int m = n - j0;
    float *Pall = sm;                                      // [kPanel + m][33]: rows of the update window, then of the panel
    float *P = Pall + kPanel * 33;                         // [m][33] staging of the panel rows (coalesced global access)
    float *vb = Pall + (((kPanel + m) * 33 + 31) & ~31);   // [2][RT * 32] published Householder vector
    float *G = vb + 2 * RT * 32;                           // [32][33]  v_i . v_j, i < j
    float *Ts = G + kPanel * (kPanel + 1);                 // [32][33]
    float *tau = Ts + kPanel * (kPanel + 1);               // [32]
    float *Vs = tau + kPanel;                              // [256][36] slab of the previous panel's vectors (fused form); later the partial sums of W
    float *Tp = Vs + 256 * 36;                             // [32][33]  previous panel's triangular factor
    float *zs = Tp + kPanel * (kPanel + 1);                // [32][33]  z = Tp^T W
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk = blockIdx.y;
    float *Amat = Abase + (long long)blockIdx.x * strideA;
    const float *A = Amat + (long long)j0 * ld + j0;

    if (prev_w > 0) {
        // ---- apply the previous panel's block reflector to this CTA's column chunk
        const int r0 = j0 - prev_w;                        // first row of the update window
        const int mu = n - r0;                             // rows of the window
        const int c0 = j0 + kPanel * chunk;                // first column of the chunk
        const int wc = min(kPanel, block_end - c0);        // columns of the chunk
        float *C = Pall + (kPanel - prev_w) * 33;          // window rows so that row prev_w of it is P's row 0
        float *Cg = Amat + (long long)r0 * ld + c0;
        const float *Vg = Vbase + (long long)blockIdx.x * strideV + (long long)r0 * ld + r0;
        for (int r = warp; r < mu; r += 32) C[r * 33 + lane] = (lane < wc) ? Cg[(long long)r * ld + lane] : 0.0f;
        for (int i = tid; i < kPanel * kPanel; i += kQrThreads) {
            const int a = i / kPanel, b = i - a * kPanel;
            Tp[a * (kPanel + 1) + b] = (a < prev_w && b < prev_w) ? Tprev_base[(long long)blockIdx.x * strideT + i] : 0.0f;
        }
        // Vp is streamed through shared memory in slabs of kSlab window rows; the next slab is
        // fetched into registers while the current one is being used, so the global-memory latency
        // of the 2 * ceil(mu / kSlab) dependent slab loads is hidden behind the arithmetic.
        // In both passes a lane works on COLUMN `lane` of the chunk and a warp on a subset of the rows,
        // so a row of Vp is read as broadcast 128-bit loads and serves all 32 columns at once (one
        // warp per column re-read every row 32 times and was bound by shared-memory bandwidth).
        constexpr int kSlab = 256, kVp = 36, kPer = kSlab * kPanel / kQrThreads;    // row pitch 36: 16-byte aligned rows
        float pre[kPer];
        auto fetch = [&](int rb) {
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                const int i = tid + q * kQrThreads, rr = i >> 5, j = i & 31;
                pre[q] = (rb + rr < mu && j < prev_w) ? Vg[(long long)(rb + rr) * ld + j] : 0.0f;
            }
        };
        auto stash = [&]() {
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                const int i = tid + q * kQrThreads;
                Vs[(i >> 5) * kVp + (i & 31)] = pre[q];
            }
        };
        // ---- W = Vp^T C.  Warp (g, h): reflector columns 8g .. 8g+7, rows h, h+8, .. of each slab.
        const int g8 = (warp >> 3) * 8, h = warp & 7;
        float wacc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) wacc[j] = 0.0f;
        fetch(0);
        for (int rb = 0; rb < mu; rb += kSlab) {
            __syncthreads();
            stash();
            __syncthreads();
            fetch(rb + kSlab < mu ? rb + kSlab : 0);       // after the last slab: the first slab of the second pass
#pragma unroll 4
            for (int k = 0; k < kSlab / 8; ++k) {
                const int rr = h + 8 * k;
                if (rb + rr < mu) {
                    const float cv = C[(rb + rr) * 33 + lane];
                    const float4 v0 = *reinterpret_cast<const float4 *>(Vs + rr * kVp + g8);
                    const float4 v1 = *reinterpret_cast<const float4 *>(Vs + rr * kVp + g8 + 4);
                    wacc[0] = fmaf(v0.x, cv, wacc[0]); wacc[1] = fmaf(v0.y, cv, wacc[1]);
                    wacc[2] = fmaf(v0.z, cv, wacc[2]); wacc[3] = fmaf(v0.w, cv, wacc[3]);
                    wacc[4] = fmaf(v1.x, cv, wacc[4]); wacc[5] = fmaf(v1.y, cv, wacc[5]);
                    wacc[6] = fmaf(v1.z, cv, wacc[6]); wacc[7] = fmaf(v1.w, cv, wacc[7]);
                }
            }
        }
        __syncthreads();                                   // the slab buffer is free: it takes the eight partial sums
        float *Wpart = Vs;                                 // [8 row groups][32][33]
#pragma unroll
        for (int j = 0; j < 8; ++j) Wpart[(h * kPanel + g8 + j) * 33 + lane] = wacc[j];
        __syncthreads();
        float *Wm = G;                                     // [32][33]; G is cleared again before the factorisation
        {
            float wsum = 0.0f;                             // W[warp][lane]
#pragma unroll
            for (int q = 0; q < 8; ++q) wsum += Wpart[(q * kPanel + warp) * 33 + lane];
            Wm[warp * 33 + lane] = wsum;
        }
        __syncthreads();
        {
            float z = 0.0f;                                // z[warp][lane] = (Tp^T W)[warp][lane]
#pragma unroll
            for (int j = 0; j < kPanel; ++j) z = fmaf(Tp[j * (kPanel + 1) + warp], Wm[j * 33 + lane], z);
            zs[warp * 33 + lane] = z;
        }
        __syncthreads();
        float zreg[kPanel];
#pragma unroll
        for (int j = 0; j < kPanel; ++j) zreg[j] = zs[j * 33 + lane];
        // ---- C -= Vp z.  Warp w: rows w, w+32, .. of each slab.
        for (int rb = 0; rb < mu; rb += kSlab) {
            __syncthreads();
            stash();
            __syncthreads();
            if (rb + kSlab < mu) fetch(rb + kSlab);
#pragma unroll 2
            for (int k = 0; k < kSlab / 32; ++k) {
                const int rr = warp + 32 * k;
                if (rb + rr < mu) {
                    float a0 = 0.0f, a1 = 0.0f;
#pragma unroll
                    for (int j = 0; j < kPanel; j += 8) {
                        const float4 v0 = *reinterpret_cast<const float4 *>(Vs + rr * kVp + j);
                        const float4 v1 = *reinterpret_cast<const float4 *>(Vs + rr * kVp + j + 4);
                        a0 = fmaf(v0.x, zreg[j], a0); a0 = fmaf(v0.y, zreg[j + 1], a0);
                        a0 = fmaf(v0.z, zreg[j + 2], a0); a0 = fmaf(v0.w, zreg[j + 3], a0);
                        a1 = fmaf(v1.x, zreg[j + 4], a1); a1 = fmaf(v1.y, zreg[j + 5], a1);
                        a1 = fmaf(v1.z, zreg[j + 6], a1); a1 = fmaf(v1.w, zreg[j + 7], a1);
                    }
                    C[(rb + rr) * 33 + lane] -= a0 + a1;
                }
            }
        }
        __syncthreads();
        if (chunk > 0) {                                   // not the new panel: write the updated chunk back and leave
            for (int r = warp; r < mu; r += 32)
                if (lane < wc) Cg[(long long)r * ld + lane] = C[r * 33 + lane];
            return;
        }
        // chunk 0: rows prev_w.. of the window are the new panel, already in P
        for (int r = warp; r < m; r += 32)
            if (lane >= w) P[r * 33 + lane] = 0.0f;
    } else {
        for (int r = warp; r < m; r += 32) P[r * 33 + lane] = (lane < w) ? A[(long long)r * ld + lane] : 0.0f;
    }
    for (int i = tid; i < 2 * kPanel * (kPanel + 1); i += kQrThreads) G[i] = 0.0f;   // G and Ts are adjacent
    __syncthreads();
    float col[RPL];
#pragma unroll
    for (int k = 0; k < RPL; ++k) {
        const int r = lane + 32 * k;
        col[k] = (r < m) ? P[r * 33 + warp] : 0.0f;
    }
    // element k of this lane's part of the column (k is a compile-time constant after unrolling)
    auto get = [&](int k) -> float {
        if (k < RPL) return col[k < RPL ? k : 0];
        const int r = lane + 32 * k;
        return r < m ? P[r * 33 + warp] : 0.0f;
    };
    auto put = [&](int k, float v) {
        if (k < RPL) { col[k < RPL ? k : 0] = v; return; }
        const int r = lane + 32 * k;
        if (r < m) P[r * 33 + warp] = v;
    };
    // Triangular factor (LAPACK slarft, forward / columnwise): T[:i, i] = -tau_i T[:i, :i] (V^T v_i)[:i].
    // Warp l owns row l of T, lane k holding T[l][k] in a register; column i is added one step after
    // its Gram entries G[:i][i] were written, by all finished warps at once (one product and one warp
    // reduction each), off the critical path of the step.
    // (The tall variants, which keep part of the panel in shared memory, have no register to spare:
    // there warp 0 fills in the column from shared memory as before.)
    constexpr bool T_IN_REGS = RS == 0;
    float trow = 0.0f;
    auto t_column_warp0 = [&](int i) {                      // whole warp; lane l computes T[l][i]
        const float ti = tau[i];
        if (lane == i) Ts[i * (kPanel + 1) + i] = ti;
        if (lane < i) {
            float a0 = 0.0f, a1 = 0.0f;
            int l = lane;
            for (; l + 1 < i; l += 2) {
                a0 = fmaf(Ts[lane * (kPanel + 1) + l], G[l * (kPanel + 1) + i], a0);
                a1 = fmaf(Ts[lane * (kPanel + 1) + l + 1], G[(l + 1) * (kPanel + 1) + i], a1);
            }
            if (l < i) a0 = fmaf(Ts[lane * (kPanel + 1) + l], G[l * (kPanel + 1) + i], a0);
            Ts[lane * (kPanel + 1) + i] = -ti * (a0 + a1);
        }
        __syncwarp();
    };
    auto t_column = [&](int i) {
        if constexpr (!T_IN_REGS) {
            if (warp == 0) t_column_warp0(i);
            return;
        }
        if (warp < i) {
            const float part = (lane >= warp && lane < i) ? trow * G[lane * (kPanel + 1) + i] : 0.0f;
            const float sum = warp_sum(part);
            if (lane == i) trow = -tau[i] * sum;
        } else if (warp == i && lane == i) {
            trow = tau[i];
        }
    };

    for (int c = 0; c < w; ++c) {
        float *vbuf = vb + (c & 1) * (RT * 32);
        if (warp == c) {
            float s4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int k = 0; k < RT; ++k) {
                const float x = get(k);
                s4[k & 3] = (lane + 32 * k > c) ? fmaf(x, x, s4[k & 3]) : s4[k & 3];
            }
            const float sigma = warp_sum((s4[0] + s4[1]) + (s4[2] + s4[3]));
            const float alpha = __shfl_sync(0xffffffffu, col[0], c);      // row c lives in lane c, slot 0
            float tc = 0.0f, scale = 0.0f;
            if (sigma != 0.0f) {
                const float beta = -copysignf(sqrtf(fmaf(alpha, alpha, sigma)), alpha);
                tc = (beta - alpha) / beta;
                scale = 1.0f / (alpha - beta);
            }
#pragma unroll
            for (int k = 0; k < RT; ++k) {
                const int r = lane + 32 * k;
                const float v = (r > c) ? get(k) * scale : (r == c ? 1.0f : 0.0f);
                put(k, v);                                  // the column now holds v_c (zeros above, one on the diagonal)
                vbuf[k * 32 + lane] = v;
            }
            if (lane == 0) tau[c] = tc;
        }
        __syncthreads();
        if (warp != c && warp < w) {
            float d4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int k = 0; k < RT; ++k) d4[k & 3] = fmaf(vbuf[k * 32 + lane], get(k), d4[k & 3]);
            const float d = warp_sum((d4[0] + d4[1]) + (d4[2] + d4[3]));
            if (warp > c) {                                 // apply H_c = I - tau v v^T to this column
                const float f = tau[c] * d;
#pragma unroll
                for (int k = 0; k < RT; ++k) put(k, fmaf(-f, vbuf[k * 32 + lane], get(k)));
            } else if (lane == 0) {
                G[warp * (kPanel + 1) + c] = d;             // v_warp . v_c
            }
        }
        // column c-1 of T: its dot products were completed before this step's barrier
        if (c >= 1) t_column(c - 1);
    }
    __syncthreads();
    t_column(w - 1);
    if constexpr (T_IN_REGS) Ts[warp * (kPanel + 1) + lane] = (lane >= warp && lane < w && warp < w) ? trow : 0.0f;
#pragma unroll
    for (int k = 0; k < RPL; ++k) {
        const int r = lane + 32 * k;
        if (r < m) P[r * 33 + warp] = col[k];
    }
    __syncthreads();
    float *V = Vbase + (long long)blockIdx.x * strideV + (long long)j0 * ld + j0;
    for (int r = warp; r < m; r += 32)
        if (lane < w) V[(long long)r * ld + lane] = P[r * 33 + lane];
    store_panel_planes(planes, P, m, w, 32);
    float *T = Tbase + (long long)blockIdx.x * strideT;
    for (int i = tid; i < kPanel * kPanel; i += kQrThreads) T[i] = Ts[(i / kPanel) * (kPanel + 1) + (i % kPanel)];
}


// ------------------------------------------------------------------------------------
// The panel kernel.  16 warps, warp w owns columns 2w and 2w+1, lane l rows l, l+32, .. of them, in registers (2 RT
// values per thread).  The 32 columns are factored in four sub-panels of eight.  Inside a sub-panel only the four warps
// that own its columns take part.  Per column step the pivot column x is published as it is, one barrier of 128 threads,
// and every warp reduces ||x||^2 together with the products of x and its own columns: one round of shuffles, no pivot
// phase that the others wait for (v = (1, x / (alpha - beta)) is a scaling that can follow).  A finished sub-panel is
// applied to the columns on its right as a block of eight: one pass over the rows for eight products per column, one
// combined reduction, a forward substitution (z_j = tau_j (w_j - sum_i<j (v_i . v_j) z_i), no triangular factor needed),
// one pass for the update - while the next sub-panel's warps, which have their own pass first, already go on factoring
// and finished columns take their products with the new vectors for the triangular factor.
//
// What bounds it is the dependent chain of 32 column steps (700 clocks each on short panels: barrier, reduction, square
// root, reciprocals).  With every warp multiplying and updating its columns in every step, and a separate pivot phase,
// a step of a tall panel took 3700 clocks.  Per launch, without / with the fused update below: 968 rows 72 / 101 -> 42 /
// 62 us, 480 rows 42 / 60 -> 28 / 41, 96 rows 25 / 32 -> 19 / 27.
//
// Fused form (prev_w > 0): the block reflector of the previous panel is applied first, C <- (I - Vp Tp^T Vp^T) C on the
// window rows j0 - prev_w .. n-1; CTA (matrix, chunk) takes 32 columns, chunk 0 is the panel itself.  Both
// products run on mma.sync (m16n8k8, tf32): every fp32 operand is split into two tf32 values, three products each,
// which keeps 2^-23 relative; at 32 columns the tile is far too small for tcgen05 and the operands come straight from
// L2 (Vp) and the shared image (C).
// ------------------------------------------------------------------------------------
static constexpr int kPw = 16, kPt = kPw * 32;            // warps and threads of a panel CTA
static constexpr int kPp = 33;                            // row pitch of the shared image: columns and 32-row groups conflict-free

// x = hi + lo to 2^-23: both rounded to tf32's 11 significant bits (half away from zero); the tensor core ignores the low
// 13 bits of an operand, so lo needs no mask.
__device__ __forceinline__ void tf32_split(float x, unsigned &hi, unsigned &lo) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi)) + 0x1000u;
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Sum of 16 values over the lanes of a warp; every lane receives all of them.
__device__ __forceinline__ void warp_sum16(float (&v)[16], int lane) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = v[i];
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1) {                       // lane bit 2h decides which half of the values it keeps
        const bool upper = (lane & (2 * h)) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float keep = upper ? x[i + h] : x[i], give = upper ? x[i] : x[i + h];
            x[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * h);
        }
    }
    x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __shfl_sync(0xffffffffu, x[0], 2 * i);   // value i sits in lanes 2i, 2i+1
}

// Products of a warp's two columns with eight vectors of the shared image (columns s0 .. s0+7; Pl: this lane's rows).
template <int RT>
__device__ __forceinline__ void dot8(const float *Pl, int s0, const float (&colA)[RT], const float (&colB)[RT], float (&z)[16], int lane) {
#pragma unroll
    for (int j = 0; j < 16; ++j) z[j] = 0.0f;
#pragma unroll
    for (int k = 0; k < RT; ++k)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float v = Pl[32 * k * kPp + s0 + j];
            z[j] = fmaf(v, colA[k], z[j]);
            z[8 + j] = fmaf(v, colB[k], z[8 + j]);
        }
    warp_sum16(z, lane);
}

template <int RT>
__global__ void __launch_bounds__(kPt, 1)
k_panel(float *__restrict__ Abase, long long strideA, int n, int ld, int j0, int w, float *__restrict__ Vbase, long long strideV,
        float *__restrict__ Tbase, long long strideT, int prev_w, const float *__restrict__ Tprev_base, int block_end, const PanelPlanes planes) {
    extern __shared__ float sm[];
    chain_wait();
    const int m = n - j0;
    float *Pall = sm;                                      // [32 + 32 RT + 32][33]: window rows above the panel, panel rows, zeros
    float *P = Pall + kPanel * kPp;
    float *part = Pall + (32 * RT + 64) * kPp;             // [8][32][33] partial sums; later the published pivot columns
    float *G = part + 8 * 32 * 33;                         // [32][33] v_i . v_j, i < j
    float *Ts = G + 32 * 33;                               // [32][33]
    float *Tp = Ts + 32 * 33, *Wm = Tp + 32 * 33, *zs = Wm + 32 * 33;
    float *tau = zs + 32 * 33;                             // [32]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, chunk = blockIdx.y;
    const int g = lane >> 2, tig = lane & 3;               // fragment coordinates of mma.m16n8k8
    float *Amat = Abase + (long long)blockIdx.x * strideA;
    float *V = Vbase + (long long)blockIdx.x * strideV;

    const int r0 = j0 - prev_w, mu = m + prev_w;           // window: first row, rows
    const int c0 = j0 + kPanel * chunk, wc = min(kPanel, prev_w > 0 ? block_end - c0 : w);
    float *C = P - prev_w * kPp;                           // window row 0
    float *Cg = Amat + (long long)r0 * ld + c0;
    if (wc == kPanel && (ld & 3) == 0 && (strideA & 3) == 0 && (reinterpret_cast<uintptr_t>(Abase) & 15) == 0) {
        // a warp takes four rows at a time, 16 bytes per lane; the four stores of a lane meet 32 different banks
#pragma unroll 8
        for (int r = 4 * warp + (lane >> 3); r < mu; r += 4 * kPw) {
            const float4 x = *reinterpret_cast<const float4 *>(Cg + (long long)r * ld + 4 * (lane & 7));
            float *dst = C + r * kPp + 4 * (lane & 7);
            dst[0] = x.x; dst[1] = x.y; dst[2] = x.z; dst[3] = x.w;
        }
    } else {
#pragma unroll 8
        for (int r = warp; r < mu; r += kPw) C[r * kPp + lane] = lane < wc ? Cg[(long long)r * ld + lane] : 0.0f;
    }
    for (int r = mu + warp; r < 32 * RT + 32 + prev_w; r += kPw) C[r * kPp + lane] = 0.0f;   // up to the end of the image
    if (prev_w > 0) {
        for (int i = tid; i < 32 * 32; i += kPt) {
            const int a = i >> 5, b = i & 31;
            Tp[a * 33 + b] = (a < prev_w && b < prev_w) ? Tprev_base[(long long)blockIdx.x * strideT + i] : 0.0f;
        }
        const float *Vg = V + (long long)r0 * ld + r0;
        const int groups = (mu + 31) >> 5;
        // ---- W = Vp^T C: k runs over the window's rows, 32 at a time; k index tig (tig + 4) of step j is row 8 tig + 2 j (+ 1),
        // which keeps the shared reads of C conflict-free
        float av[4][8];
        auto fetch_v = [&](int gr) {
            if (gr >= groups) return;
            const float *vg = Vg + (long long)(32 * gr + 8 * tig) * ld + g;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int row = 32 * gr + 8 * tig + 2 * j + (q >> 2);
                    av[j][q] = (row < mu && g + 8 * (q & 3) < prev_w) ? vg[(2 * j + (q >> 2)) * ld + 8 * (q & 3)] : 0.0f;
                }
        };
        fetch_v(warp);
        __syncthreads();
        float acc[2][4][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0f;
        for (int gr = warp; gr < groups; gr += kPw) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                unsigned ah[2][4], al[2][4], bh[4][2], bl[4][2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {              // a0: (g, tig), a1: (g + 8, tig), a2: (g, tig + 4), a3: (g + 8, tig + 4)
                    tf32_split(av[j][2 * i], ah[i][0], al[i][0]);
                    tf32_split(av[j][2 * i + 1], ah[i][1], al[i][1]);
                    tf32_split(av[j][4 + 2 * i], ah[i][2], al[i][2]);
                    tf32_split(av[j][4 + 2 * i + 1], ah[i][3], al[i][3]);
                }
                const float *cr = C + (32 * gr + 8 * tig + 2 * j) * kPp + g;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    tf32_split(cr[8 * t], bh[t][0], bl[t][0]);
                    tf32_split(cr[kPp + 8 * t], bh[t][1], bl[t][1]);
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) { mma_tf32(acc[0][t], al[0], bh[t]); mma_tf32(acc[1][t], al[1], bh[t]); }
#pragma unroll
                for (int t = 0; t < 4; ++t) { mma_tf32(acc[0][t], ah[0], bl[t]); mma_tf32(acc[1][t], ah[1], bl[t]); }
#pragma unroll
                for (int t = 0; t < 4; ++t) { mma_tf32(acc[0][t], ah[0], bh[t]); mma_tf32(acc[1][t], ah[1], bh[t]); }
            }
            fetch_v(gr + kPw);
        }
        // sum of the warps' partial results: eight leave theirs, the other eight add, the eight sums are added by all
        float *mine = part + (warp & 7) * (32 * 33) + g * 33 + 2 * tig;
#pragma unroll
        for (int half = 1; half >= 0; --half) {
            if ((warp >> 3) == half) {
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int t = 0; t < 4; ++t)
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            float *d = mine + (16 * i + 8 * (q >> 1)) * 33 + 8 * t + (q & 1);
                            if (half) *d = acc[i][t][q]; else *d += acc[i][t][q];
                        }
            }
            __syncthreads();
        }
        for (int jr = warp; jr < 32; jr += kPw) {
            float s = 0.0f;
#pragma unroll
            for (int q = 0; q < 8; ++q) s += part[q * (32 * 33) + jr * 33 + lane];
            Wm[jr * 33 + lane] = s;
        }
        __syncthreads();
        for (int jr = warp; jr < 32; jr += kPw) {           // z = Tp^T W
            float z0 = 0.0f, z1 = 0.0f;
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                z0 = fmaf(Tp[j * 33 + jr], Wm[j * 33 + lane], z0);
                z1 = fmaf(Tp[(j + 1) * 33 + jr], Wm[(j + 1) * 33 + lane], z1);
            }
            zs[jr * 33 + lane] = z0 + z1;
        }
        __syncthreads();
        // ---- C -= Vp z, 32 rows at a time: fragment row g (g + 8) of tile rt is row 4 g + 2 rt (+ 1)
        float zr[4][4][2];                                  // z fragments: k-step, column tile
#pragma unroll
        for (int kb = 0; kb < 4; ++kb)
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                zr[kb][t][0] = zs[(8 * kb + tig) * 33 + 8 * t + g];
                zr[kb][t][1] = zs[(8 * kb + tig + 4) * 33 + 8 * t + g];
            }
        for (int gr = warp; gr < groups; gr += kPw) {
            const int row = 32 * gr + 4 * g;
            const float *vg = Vg + (long long)row * ld + tig;
            float up[2][4][4], a[2][4];
#pragma unroll
            for (int rt = 0; rt < 2; ++rt)
#pragma unroll
                for (int t = 0; t < 4; ++t)
#pragma unroll
                    for (int q = 0; q < 4; ++q) up[rt][t][q] = 0.0f;
            auto fetch_a = [&](int kb) {
#pragma unroll
                for (int rt = 0; rt < 2; ++rt)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int dr = 2 * rt + (q & 1), dc = 8 * kb + 4 * (q >> 1);
                        a[rt][q] = (row + dr < mu && tig + dc < prev_w) ? vg[dr * ld + dc] : 0.0f;
                    }
            };
            fetch_a(0);
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                unsigned ah[2][4], al[2][4], bh[4][2], bl[4][2];
#pragma unroll
                for (int rt = 0; rt < 2; ++rt)
#pragma unroll
                    for (int q = 0; q < 4; ++q) tf32_split(a[rt][q], ah[rt][q], al[rt][q]);
                if (kb < 3) fetch_a(kb + 1);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    tf32_split(zr[kb][t][0], bh[t][0], bl[t][0]);
                    tf32_split(zr[kb][t][1], bh[t][1], bl[t][1]);
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) { mma_tf32(up[0][t], al[0], bh[t]); mma_tf32(up[1][t], al[1], bh[t]); }
#pragma unroll
                for (int t = 0; t < 4; ++t) { mma_tf32(up[0][t], ah[0], bl[t]); mma_tf32(up[1][t], ah[1], bl[t]); }
#pragma unroll
                for (int t = 0; t < 4; ++t) { mma_tf32(up[0][t], ah[0], bh[t]); mma_tf32(up[1][t], ah[1], bh[t]); }
            }
#pragma unroll
            for (int rt = 0; rt < 2; ++rt) {
                float *cr = C + (row + 2 * rt) * kPp + 2 * tig;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    cr[8 * t] -= up[rt][t][0];
                    cr[8 * t + 1] -= up[rt][t][1];
                    cr[kPp + 8 * t] -= up[rt][t][2];
                    cr[kPp + 8 * t + 1] -= up[rt][t][3];
                }
            }
        }
        __syncthreads();
        if (chunk > 0) {                                   // not the new panel: write the updated chunk back and leave
            chain_release();
#pragma unroll 4
            for (int r = warp; r < mu; r += kPw)
                if (lane < wc) Cg[(long long)r * ld + lane] = C[r * kPp + lane];
            return;
        }
        if (w < kPanel)
            for (int r = warp; r < m; r += kPw)
                if (lane >= w) P[r * kPp + lane] = 0.0f;
    }
    for (int i = tid; i < 2 * 32 * 33; i += kPt) G[i] = 0.0f;   // G and Ts are adjacent
    if (tid < 32) tau[tid] = 0.0f;
    __syncthreads();

    // ---- factorisation
    const int cA = 2 * warp, cB = cA + 1;
    float colA[RT], colB[RT];
#pragma unroll
    for (int k = 0; k < RT; ++k) {
        colA[k] = P[(lane + 32 * k) * kPp + cA];
        colB[k] = P[(lane + 32 * k) * kPp + cB];
    }
    const float *Pl = P + lane * kPp;                      // this lane's rows
#pragma unroll 1
    for (int sp = 0; sp < 4 && 8 * sp < w; ++sp) {
        if ((warp >> 2) == sp) {
            const int end = min(8 * sp + 8, w);
            float *xb = part + lane;                          // [2][RT * 32] the pivot column as it is, double-buffered
            float scA = 0.0f, scB = 0.0f;                     // scalings of this warp's finished pivots
            if (cA == 8 * sp) {
#pragma unroll
                for (int k = 0; k < RT; ++k) xb[32 * k] = colA[k];
            }
#pragma unroll 1
            for (int c = 8 * sp; c < end; ++c) {
                const float *xc = xb + (c & 1) * (32 * RT);
                asm volatile("bar.sync 1, 128;" ::: "memory");
                // one round of reductions: the pivot's norm (every warp for itself) and the products with both columns
                float s2[2] = {0.0f, 0.0f}, a2[2] = {0.0f, 0.0f}, b2[2] = {0.0f, 0.0f};
#pragma unroll
                for (int k = 0; k < RT; ++k) {
                    float x = xc[32 * k];
                    if (k == 0) x = lane > c ? x : 0.0f;
                    s2[k & 1] = fmaf(x, x, s2[k & 1]);
                    a2[k & 1] = fmaf(x, colA[k], a2[k & 1]);
                    b2[k & 1] = fmaf(x, colB[k], b2[k & 1]);
                }
                const float alpha = part[(c & 1) * (32 * RT) + c];
                const float eA = __shfl_sync(0xffffffffu, colA[0], c), eB = __shfl_sync(0xffffffffu, colB[0], c);   // row c: lane c, slot 0
                float sigma = s2[0] + s2[1], dA = a2[0] + a2[1], dB = b2[0] + b2[1];
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) {
                    sigma += __shfl_xor_sync(0xffffffffu, sigma, off);
                    dA += __shfl_xor_sync(0xffffffffu, dA, off);
                    dB += __shfl_xor_sync(0xffffffffu, dB, off);
                }
                // tau = (beta - alpha) / beta, v = (1, scale x): tau * scale = -1 / beta, so the update waits for two
                // reciprocals side by side and not for a division
                float rb = 0.0f, scale = 0.0f, diff = 0.0f;
                if (sigma != 0.0f) {
                    const float beta = -copysignf(sqrtf(fmaf(alpha, alpha, sigma)), alpha);
                    diff = beta - alpha;
                    rb = 1.0f / beta;
                    scale = -1.0f / diff;
                }
                const float tc = diff * rb;
                dA = fmaf(scale, dA, eA);                     // v . column
                dB = fmaf(scale, dB, eB);
                __syncwarp();                                 // x is read again: RT values kept from the products would spill
                if (cB > c) {                                 // at least column B is updated (warp-uniform)
                    const float fA = cA > c ? tc * dA : 0.0f, fB = tc * dB;
                    const float hA = cA > c ? -rb * dA : 0.0f, hB = -rb * dB;
                    const float x0 = xc[0];
                    colA[0] = lane > c ? fmaf(-hA, x0, colA[0]) : (lane == c ? colA[0] - fA : colA[0]);
                    colB[0] = lane > c ? fmaf(-hB, x0, colB[0]) : (lane == c ? colB[0] - fB : colB[0]);
#pragma unroll
                    for (int k = 1; k < RT; ++k) {
                        const float x = xc[32 * k];
                        colA[k] = fmaf(-hA, x, colA[k]);
                        colB[k] = fmaf(-hB, x, colB[k]);
                    }
                    if (c + 1 < end && warp == ((c + 1) >> 1)) {      // the next pivot
                        float *xn = xb + ((c + 1) & 1) * (32 * RT);
#pragma unroll
                        for (int k = 0; k < RT; ++k) xn[32 * k] = cA == c + 1 ? colA[k] : colB[k];
                    }
                }
                // finished columns are still unscaled: v_col . v_c = scale_col (scale_c x_col . x + x_col[c])
                if (cA < c && lane == 0) G[cA * 33 + c] = scA * dA;
                if (cB < c && lane == 0) G[cB * 33 + c] = scB * dB;
                if (cA == c) scA = scale;
                if (cB == c) scB = scale;
                if (warp == (c >> 1) && lane == 0) tau[c] = tc;
            }
            if (cA < end) {                                   // the pivots become v
                float *pub = P + lane * kPp + cA;
#pragma unroll
                for (int k = 0; k < RT; ++k) {
                    colA[k] *= scA;
                    if (k == 0) colA[0] = lane > cA ? colA[0] : (lane == cA ? 1.0f : 0.0f);
                    pub[32 * k * kPp] = colA[k];
                    if (cB < end) {
                        colB[k] *= scB;
                        if (k == 0) colB[0] = lane > cB ? colB[0] : (lane == cB ? 1.0f : 0.0f);
                        pub[32 * k * kPp + 1] = colB[k];
                    }
                }
            }
        }
        __syncthreads();                                      // the sub-panel's vectors, tau and products are published
        // the next sub-panel's warps have shared memory to themselves for their pass; the others follow beside its column steps
        const bool next = (warp >> 2) == sp + 1;
        const int s0 = 8 * sp;
        float z[16];                                          // [column A / B][vector]
        if (sp < 3 && !next) asm volatile("bar.sync 3, 512;" ::: "memory");
        if (warp >= 4 * sp + 4 && cA < w) {
            dot8<RT>(Pl, s0, colA, colB, z, lane);
            __syncwarp();                                     // the vectors are read again (8 RT values kept would spill)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float a = z[j], b = z[8 + j];
#pragma unroll
                for (int i = 0; i < j; ++i) {
                    const float gij = G[(s0 + i) * 33 + s0 + j];
                    a = fmaf(-gij, z[i], a);
                    b = fmaf(-gij, z[8 + i], b);
                }
                const float tj = tau[s0 + j];
                z[j] = tj * a;
                z[8 + j] = tj * b;
            }
#pragma unroll
            for (int k = 0; k < RT; ++k)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float v = Pl[32 * k * kPp + s0 + j];
                    colA[k] = fmaf(-z[j], v, colA[k]);
                    colB[k] = fmaf(-z[8 + j], v, colB[k]);
                }
        } else if (warp < 4 * sp) {                           // finished columns: their products with the new vectors
            dot8<RT>(Pl, s0, colA, colB, z, lane);
            if (lane == 0) {
#pragma unroll
                for (int j = 0; j < 8; ++j) { G[cA * 33 + s0 + j] = z[j]; G[cB * 33 + s0 + j] = z[8 + j]; }
            }
        }
        if (next) asm volatile("bar.arrive 3, 512;" ::: "memory");
    }
    chain_release();
    __syncthreads();
    // ---- triangular factor from V^T V and tau (LAPACK slarft): four 8 x 8 blocks, then -T1 (G12 T2) for the off-diagonal
    // blocks of 8 and of 16.  Eight warps; the others store V meanwhile.  (One warp running down 32 columns took 5600 clocks.)
    if (warp < 8) {
        auto sync8 = [] { asm volatile("bar.sync 2, 256;" ::: "memory"); };
        if (warp < 4 && lane < 8) {
            const int b = 8 * warp;
            float t[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float x = 0.0f;
#pragma unroll
                for (int k = 0; k < i; ++k) x = fmaf(t[k], G[(b + k) * 33 + b + i], x);   // t[k] is zero for k < lane
                const float ti = tau[b + i];
                t[i] = lane < i ? -ti * x : (lane == i ? ti : 0.0f);
                Ts[(b + lane) * 33 + b + i] = t[i];
            }
        }
        sync8();
        const int p = 16 * (tid >> 6), pr = p + ((tid >> 3) & 7), pc = p + 8 + (tid & 7);
        if (tid < 128) {                                      // pairs of 8: Wm = G12 T2
            float x = 0.0f;
#pragma unroll
            for (int k = 0; k < 8; ++k) x = fmaf(G[pr * 33 + p + 8 + k], Ts[(p + 8 + k) * 33 + pc], x);
            Wm[pr * 33 + pc] = x;
        }
        sync8();
        if (tid < 128) {
            float x = 0.0f;
#pragma unroll
            for (int k = 0; k < 8; ++k) x = fmaf(Ts[pr * 33 + p + k], Wm[(p + k) * 33 + pc], x);
            Ts[pr * 33 + pc] = -x;
        }
        sync8();
        const int r = tid >> 4, c = 16 + (tid & 15);          // 256 threads: the 16 x 16 block
        float x = 0.0f, y = 0.0f;
#pragma unroll
        for (int k = 0; k < 16; ++k) x = fmaf(G[r * 33 + 16 + k], Ts[(16 + k) * 33 + c], x);
        Wm[r * 33 + c] = x;
        sync8();
#pragma unroll
        for (int k = 0; k < 16; ++k) y = fmaf(Ts[r * 33 + k], Wm[k * 33 + c], y);
        Ts[r * 33 + c] = -y;
        sync8();
        float *T = Tbase + (long long)blockIdx.x * strideT;
        for (int i = tid; i < kPanel * kPanel; i += 256) {
            const int a = i >> 5, b = i & 31;
            T[i] = (a < w && b < w) ? Ts[a * 33 + b] : 0.0f;
        }
    }
    float *Vo = V + (long long)j0 * ld + j0;
#pragma unroll 4
    for (int r = warp; r < m; r += kPw)
        if (lane < w) Vo[(long long)r * ld + lane] = P[r * kPp + lane];
    store_panel_planes(planes, P, m, w, kPw);
}

template <int RT>
static int launch_panel(float *A, long long strideA, int n, int ld, int count, int j0, int w, float *V, long long strideV, float *T, long long strideT,
                        cudaStream_t s, int prev_w, const float *Tprev, int block_end, const PanelPlanes &planes, bool chained) {
    const size_t smem = sizeof(float) * ((size_t)(32 * RT + 64) * kPp + 8 * 32 * 33 + 5 * 32 * 33 + 32);
    static PerDeviceOnce attr_set;
    const int dev = current_device();
    if (attr_set.pending(dev)) {
        if (cudaFuncSetAttribute(k_panel<RT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return record(QT_ERR_LAUNCH);
        attr_set.mark(dev);
    }
    const int chunks = prev_w > 0 ? (block_end - j0 + kPanel - 1) / kPanel : 1;
    if (launch_chained(k_panel<RT>, dim3(count, chunks), kPt, smem, s, chained, A, strideA, n, ld, j0, w, V, strideV, T, strideT, prev_w, Tprev, block_end,
                       planes) != cudaSuccess) { cudaGetLastError(); return record(QT_ERR_LAUNCH); }
    count_launch(1);
    return check_launch();
}

template <int RPL, int RS>
static int launch_panel_rpl(float *A, long long strideA, int n, int ld, int count, int j0, int w,
                            float *V, long long strideV, float *T, long long strideT, cudaStream_t s,
                            int prev_w, const float *Tprev, int block_end, const PanelPlanes &planes) {
    const int m = n - j0;
    const size_t smem = sizeof(float) * ((size_t)(((kPanel + m) * 33 + 31) & ~31) + 2 * (RPL + RS) * 32 + 2 * kPanel * (kPanel + 1) + kPanel +
                                         256 * 36 + kPanel * (kPanel + 1) + kPanel * (kPanel + 1));
    static PerDeviceOnce attr_set;                         // function attributes are per device
    const int dev = current_device();
    if (attr_set.pending(dev)) {
        if (cudaFuncSetAttribute(k_householder_panel<RPL, RS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
            return record(QT_ERR_LAUNCH);
        attr_set.mark(dev);
    }
    if (smem > 227 * 1024) return record(QT_ERR_UNSUPPORTED);
    const int chunks = prev_w > 0 ? (block_end - j0 + kPanel - 1) / kPanel : 1;
    dim3 grid(count, chunks);
    k_householder_panel<RPL, RS><<<grid, kQrThreads, smem, s>>>(A, strideA, n, ld, j0, w, V, strideV, T, strideT, prev_w, Tprev, block_end, planes);
    count_launch(1);
    return check_launch();
}

int launch_householder_panel(float *A, long long strideA, int n, int ld, int count, int j0, int w,
                             float *V, long long strideV, float *T, long long strideT, cudaStream_t s,
                             int prev_w, const float *Tprev, int block_end,
                             void *planes_hi, void *planes_lo, long long ldp, long long strideP, int plane_col, int rows_above, int plane_exp, bool chained) {
    const PanelPlanes planes{static_cast<__half *>(planes_hi), static_cast<__half *>(planes_lo), ldp, strideP, plane_col, rows_above,
                             ldexpf(1.0f, plane_exp)};
    if (ld < n || n <= 0 || count < 0 || j0 < 0 || j0 >= n || w <= 0 || w > kPanel || j0 + w > n) return record(QT_ERR_ARG);
    if (!A || !V || !T) return record(QT_ERR_ARG);
    if (prev_w < 0 || prev_w > kPanel || prev_w > j0) return record(QT_ERR_ARG);
    if (prev_w > 0 && (!Tprev || block_end < j0 + w || block_end > n || block_end - j0 > 4 * kPanel)) return record(QT_ERR_ARG);
    if (count == 0) return record(QT_OK);
    if (count > 65535) return record(QT_ERR_UNSUPPORTED);
    const int rows_per_lane = (n - j0 + 31) / 32;
    if (rows_per_lane > kMaxRowsPerLane) return record(QT_ERR_UNSUPPORTED);
#define QT_ARGS A, strideA, n, ld, count, j0, w, V, strideV, T, strideT, s, prev_w, Tprev, block_end, planes
    if (!g_panel_blocked) {
        if (rows_per_lane <= 20) return launch_panel_rpl<20, 0>(QT_ARGS);
        return launch_panel_rpl<24, 14>(QT_ARGS);
    }
    // rows per lane are rounded up to a multiple of four: the factorisation's time goes with them
    if (rows_per_lane <= 4) return launch_panel<4>(QT_ARGS, chained);
    if (rows_per_lane <= 8) return launch_panel<8>(QT_ARGS, chained);
    if (rows_per_lane <= 12) return launch_panel<12>(QT_ARGS, chained);
    if (rows_per_lane <= 16) return launch_panel<16>(QT_ARGS, chained);
    if (rows_per_lane <= 20) return launch_panel<20>(QT_ARGS, chained);
    if (rows_per_lane <= 24) return launch_panel<24>(QT_ARGS, chained);
    if (rows_per_lane <= 28) return launch_panel<28>(QT_ARGS, chained);
    if (rows_per_lane <= 32) return launch_panel<32>(QT_ARGS, chained);
    return launch_panel<38>(QT_ARGS, chained);
#undef QT_ARGS
}

// Triangular factor of an outer block of up to four panels from the panels' own factors and
// the Gram matrix G = Vo^T Vo of the block's Householder vectors (LAPACK larft on blocks, by halves):
//     T = [T1, -T1 (G12 T2); 0, T2],   first for the two pairs of 32 columns, then for the pair of 64.
// One CTA per matrix; everything is padded with zeros to 128 columns in shared memory and T is written out whole (zeros
// below the diagonal blocks).  Bound by latency and by shared-memory wavefronts: the chain is two products of 32^3 and two of
// 64^3 where panel after panel took three pairs of products that grew with the columns done, and a warp's tile of 8 rows
// x 16 columns reads four k of a row and of four columns at a time, conflict-free: 5 wavefronts per 4 x 128
// multiply-adds (one operand and one wavefront per multiply-add before).  28 -> 14 us.
static constexpr int kMergeMax = 128, kMergeP = 132;         // row pitch: 16-byte rows, 8 rows meet 32 banks

// out[i][j] (+)= sgn * sum over l in [l0, l1) of A[i][l] B[l][j], for this lane's row i and columns j .. j+3
__device__ __forceinline__ float4 merge_dot(const float *a, const float *b, int l0, int l1) {
    float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int l = l0; l < l1; l += 4) {
        const float4 x = *reinterpret_cast<const float4 *>(a + l);
        const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 y = *reinterpret_cast<const float4 *>(b + (l + q) * kMergeP);
            r.x = fmaf(xs[q], y.x, r.x); r.y = fmaf(xs[q], y.y, r.y);
            r.z = fmaf(xs[q], y.z, r.z); r.w = fmaf(xs[q], y.w, r.w);
        }
    }
    return r;
}

__global__ void __launch_bounds__(1024)
k_merge_t(const float *__restrict__ Gbase, long long ldg, long long strideG,
          const float *__restrict__ Tp_base, long long strideTp, int wo,
          float *__restrict__ Tbase, long long strideT,
          __half *__restrict__ hi, __half *__restrict__ lo, long long ldp, long long strideP, int *__restrict__ exp_out, int target) {
    extern __shared__ __align__(16) float merge_sm[];
    chain_wait();
    float *Ts = merge_sm, *Gs = Ts + kMergeMax * kMergeP, *red = Gs + kMergeMax * kMergeP;
    const float *G = Gbase + (long long)blockIdx.x * strideG;
    const float *Tp = Tp_base + (long long)blockIdx.x * strideTp;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the panels' factors on the diagonal, zeros elsewhere; the Gram matrix's blocks above the diagonal
    const bool vec_g = (ldg & 3) == 0 && (strideG & 3) == 0 && (reinterpret_cast<uintptr_t>(Gbase) & 15) == 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int e = tid + 1024 * u, i = e >> 5, j = (e & 31) * 4;
        float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f), g = t;
        float ts[4] = {0.0f, 0.0f, 0.0f, 0.0f}, gs[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if ((i >> 5) == (j >> 5) && i < wo) {
            const float *src = Tp + (long long)(i >> 5) * kPanel * kPanel + (i & 31) * kPanel + (j & 31);
#pragma unroll
            for (int q = 0; q < 4; ++q) if (j + q < wo) ts[q] = src[q];
        }
        if ((j >> 5) > (i >> 5) && i < wo) {
            const float *src = G + (long long)i * ldg + j;
            if (vec_g && j + 3 < wo) { g = __ldg(reinterpret_cast<const float4 *>(src)); gs[0] = g.x; gs[1] = g.y; gs[2] = g.z; gs[3] = g.w; }
            else {
#pragma unroll
                for (int q = 0; q < 4; ++q) if (j + q < wo) gs[q] = __ldg(src + q);
            }
        }
        t = make_float4(ts[0], ts[1], ts[2], ts[3]);
        g = make_float4(gs[0], gs[1], gs[2], gs[3]);
        *reinterpret_cast<float4 *>(Ts + i * kMergeP + j) = t;
        *reinterpret_cast<float4 *>(Gs + i * kMergeP + j) = g;
    }
    __syncthreads();
    // pairs of 32 columns at b = 0 and 64: eight warps each; the intermediate product lies below G's diagonal
    const int b = 64 * (warp >> 3), w8 = warp & 7;
    const int i1 = 8 * (w8 & 3) + (lane >> 2), j1 = 16 * (w8 >> 2) + 4 * (lane & 3);
    const bool one = warp < 16 && b + 32 < wo;
    if (one) *reinterpret_cast<float4 *>(Gs + (b + 32 + i1) * kMergeP + b + j1) =
                 merge_dot(Gs + (b + i1) * kMergeP + b + 32, Ts + (b + 32) * kMergeP + b + 32 + j1, 0, 16 * (w8 >> 2) + 16);   // T2 is upper triangular
    __syncthreads();
    if (one) {
        const float4 r = merge_dot(Ts + (b + i1) * kMergeP + b, Gs + (b + 32) * kMergeP + b + j1, 8 * (w8 & 3), 32);           // and T1
        *reinterpret_cast<float4 *>(Ts + (b + i1) * kMergeP + b + 32 + j1) = make_float4(-r.x, -r.y, -r.z, -r.w);
    }
    __syncthreads();
    chain_release();
    if (wo > 64) {                                            // the pair of 64: all warps
        const int i2 = 8 * (warp & 7) + (lane >> 2), j2 = 16 * (warp >> 3) + 4 * (lane & 3);
        *reinterpret_cast<float4 *>(Gs + (64 + i2) * kMergeP + j2) = merge_dot(Gs + i2 * kMergeP + 64, Ts + 64 * kMergeP + 64 + j2, 0, 16 * (warp >> 3) + 16);
        __syncthreads();
        const float4 r = merge_dot(Ts + i2 * kMergeP, Gs + 64 * kMergeP + j2, 8 * (warp & 7), 64);
        *reinterpret_cast<float4 *>(Ts + i2 * kMergeP + 64 + j2) = make_float4(-r.x, -r.y, -r.z, -r.w);
        __syncthreads();
    }
    if (Tbase) {
        float *T = Tbase + (long long)blockIdx.x * strideT;
        for (int i = warp; i < wo; i += 32)
            for (int j = lane; j < wo; j += 32) T[(long long)i * wo + j] = Ts[i * kMergeP + j];
    }
    if (!hi) return;
    // scaled fp16 planes of T (the operand of the products that follow), exponent from the largest magnitude
    float v[2][8], am = 0.0f;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int e = tid + 1024 * u, i = e >> 4, j = (e & 15) * 8;
#pragma unroll
        for (int q = 0; q < 8; q += 4) {
            const float4 x = *reinterpret_cast<const float4 *>(Ts + i * kMergeP + j + q);
            v[u][q] = x.x; v[u][q + 1] = x.y; v[u][q + 2] = x.z; v[u][q + 3] = x.w;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) am = fmaxf(am, fabsf(v[u][q]));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, off));
    if (lane == 0) red[warp] = am;
    __syncthreads();
    am = red[lane];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, off));
    const int e_out = exponent_for(am, target);
    if (tid == 0) exp_out[blockIdx.x] = e_out;
    const float two_e = exp2f((float)e_out);
    hi += (long long)blockIdx.x * strideP;
    lo += (long long)blockIdx.x * strideP;
    const bool vec_p = ((ldp | strideP) & 7) == 0 && ((reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 15) == 0;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int e = tid + 1024 * u, i = e >> 4, j = (e & 15) * 8;
        if (i >= wo || j >= wo) continue;
        __half h[8], l[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float x = fminf(fmaxf(v[u][q] * two_e, -65000.0f), 65000.0f);
            h[q] = __float2half_rn(x);
            l[q] = __float2half_rn(x - __half2float(h[q]));
        }
        __half *dh = hi + (long long)i * ldp + j, *dl = lo + (long long)i * ldp + j;
        if (vec_p && j + 8 <= wo) {
            auto word = [](const __half *p) { return (unsigned)__half_as_ushort(p[0]) | ((unsigned)__half_as_ushort(p[1]) << 16); };
            *reinterpret_cast<uint4 *>(dh) = make_uint4(word(h), word(h + 2), word(h + 4), word(h + 6));
            *reinterpret_cast<uint4 *>(dl) = make_uint4(word(l), word(l + 2), word(l + 4), word(l + 6));
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) if (j + q < wo) { dh[q] = h[q]; dl[q] = l[q]; }
        }
    }
}

int launch_merge_t(const float *G, long long ldg, long long strideG, const float *Tp, long long strideTp, int wo, int count,
                   float *T, long long strideT, cudaStream_t s, void *hi, void *lo, long long ldp, long long strideP, int *exp_out, int target, bool chained) {
    if (wo <= 0 || wo > kMergeMax || count < 0 || ldg < wo) return record(QT_ERR_ARG);
    if (!G || !Tp || (!T && !hi) || (hi && (!lo || !exp_out || ldp < wo))) return record(QT_ERR_ARG);
    if (count == 0) return record(QT_OK);
    constexpr size_t smem = sizeof(float) * (2 * kMergeMax * kMergeP + 32);
    static PerDeviceOnce attr_set;
    const int dev = current_device();
    if (attr_set.pending(dev)) {
        if (cudaFuncSetAttribute(k_merge_t, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return record(QT_ERR_LAUNCH);
        attr_set.mark(dev);
    }
    if (launch_chained(k_merge_t, count, 1024, smem, s, chained, G, ldg, strideG, Tp, strideTp, wo, T, strideT, static_cast<__half *>(hi),
                       static_cast<__half *>(lo), ldp, strideP, exp_out, target) != cudaSuccess) { cudaGetLastError(); return record(QT_ERR_LAUNCH); }
    count_launch(1);
    return check_launch();
}

}  // namespace qt
