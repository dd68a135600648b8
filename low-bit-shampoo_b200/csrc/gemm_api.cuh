// Argument structures and launchers of the tensor-core products, for the host-side orchestrations of the library.
#pragma once
#include "qt_common.cuh"

namespace qt {

// A product operand that lives as 4-bit blockwise state: matrix b of the product is state slot
// slots[b] (null: b); its plane exponent is a_exp[b] / b_exp[b] of GemmParams.
struct QOperand {
    const unsigned char *codes; const float *absmax, *diag; const int *slots;
    long long stride_codes, stride_absmax, stride_diag;                   // per slot: bytes, floats, floats
    int n, nb;                                                            // order of the state matrices, blocks per row
};

struct GemmArgs {
    const void *Ahi, *Alo; long long lda, strideA; int a_mn;
    const void *Bhi, *Blo; long long ldb, strideB; int b_mn;
    int M, N, K, batch; float alpha, beta;
    const float *C; long long ldc, strideC;
    float *D; long long ldd, strideD;
    void *Dhi, *Dlo; long long ldp, strideP;
};

// Optional extras of a product (all pointers device memory, any of them may be null).
struct GemmExtras {
    void *Dmid = nullptr;                                   // middle result plane (three-plane products)
    void *Thi = nullptr, *Tmid = nullptr, *Tlo = nullptr;   // t_c0 * I + t_c1 * result, three planes (pitch of the result planes)
    float t_c0 = 0.0f, t_c1 = 0.0f;
    float *maxdev = nullptr;                                // per matrix max |result - I|
    const int *a_slot = nullptr, *b_slot = nullptr, *d_slot = nullptr;
    const int *active = nullptr;
    int a_entries = 0, b_entries = 0;                       // matrices in A's / B's storage (0: batch)
    // scaled fp16 planes (two-plane products only)
    int f16 = 0;
    const int *a_exp = nullptr, *b_exp = nullptr; int ab_exp0 = 0;
    const int *out_exp = nullptr; int *out_exp_w = nullptr; int out_exp0 = 0, out_rel = 0;
    int kc = 0;                                             // k-blocks per accumulation chain (0: one chain)
    // operands straight from 4-bit state (see QOperand); codes == nullptr: from planes
    QOperand aq = {nullptr, nullptr, nullptr, nullptr, 0, 0, 0, 0, 0}, bq = {nullptr, nullptr, nullptr, nullptr, 0, 0, 0, 0, 0};
    const float *oq_code = nullptr;
    int max_ctas = 0;                                       // > 0: cap of the persistent grid (SMs left to kernels on other streams)
    int c_follows_d = 0;                                    // C indexed through d_slot like the outputs
    int sym = 0;                                            // the result is symmetric (M == N): tiles on and above the diagonal, mirrored
    int chained = 0;                                        // the launch may overlap the end of its predecessor (see launch_chained)
    float *amax_out = nullptr;                              // per output entry: max |result| (atomic max; zeroed by the caller)
    float *cd_part = nullptr;                               // column sums of result * C instead of a stored result: per matrix
                                                            // [4 * ceil(M / 128)][N] partial sums (two planes)
};

// 4-bit state operands of the quantizing variant (all device pointers; see GemmParams).
struct QuantStateArgs {
    const float *code;
    const unsigned char *q_in; const float *absmax_in, *diag_in;
    unsigned char *q_out; float *absmax_out, *diag_out;
    long long stride_codes, stride_absmax, stride_diag;
};


// a.Ahi/Alo (+ Amid/Bmid for three planes: order hi, mid, lo).  With `qs` the result (and the C
// operand, if qs->q_in) is 4-bit state instead of a.C / a.D.
int launch_gemm_planes(const GemmArgs &a, const void *Amid, const void *Bmid, cudaStream_t s, const QuantStateArgs *qs,
                       const GemmExtras *ex = nullptr);
int launch_split_f16(const float *X, long long ldx, long long strideX, int rows, int cols, int batch,
                     const long long *index, long long stride_index, const float *scale, long long stride_scale,
                     float *amax, int compute_amax, const int *exp_in, int target_or_exp0, int *exp_out,
                     void *hi, void *lo, long long ldp, long long strideP, cudaStream_t s);

}  // namespace qt
