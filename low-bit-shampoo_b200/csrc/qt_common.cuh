// Shared declarations of libqtensor_b200: status codes, stream / error bookkeeping and
// the launcher prototypes that abi.cu forwards to.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include "../../include/qtensor_b200.h"

namespace qt {

// Thread-local state behind qt_set_stream / qt_last_error.
cudaStream_t current_stream();
void set_current_stream(cudaStream_t s);
int record(int status);          // stores status as this thread's last error and returns it
void count_launch(int n);        // adds n to the process-wide kernel launch counter
int check_launch();              // cudaGetLastError -> QT_OK / QT_ERR_LAUNCH (recorded)

// Per-device bookkeeping: function attributes (cudaFuncSetAttribute) and the SM count belong to
// one device, and a process may drive several.  Ordinals at or above kMaxDevices are refused.
static constexpr int kMaxDevices = 64;
int current_device();            // ordinal of the calling thread's current device, or -1
int device_sm_count();           // SM count of the current device (cached per device; 148 if unknown)
// One flag per device.  pending() is true until mark() has been called for that device; a
// race between two first callers only repeats an idempotent set-up.
struct PerDeviceOnce {
    volatile unsigned char done[kMaxDevices];
    bool pending(int dev) const { return dev < 0 || dev >= kMaxDevices || !done[dev]; }
    void mark(int dev) { if (dev >= 0 && dev < kMaxDevices) done[dev] = 1; }
};

inline bool valid_blocksize(int bs) {
    return bs == 64 || bs == 128 || bs == 256 || bs == 512 || bs == 1024 || bs == 2048;
}

struct QuantArgs {
    const void *A; int a_dtype; long long strideA;          // elements
    const float *code;
    int n, count, bs, bits;
    float *absmax; long long stride_absmax;
    float *diag; long long stride_diag;                     // diag == nullptr: plain variant
    unsigned char *out; long long stride_out;               // bytes
};

struct DequantArgs {
    const unsigned char *A; long long strideA;              // bytes
    const float *code;
    int n, count, bs, bits;
    const float *absmax; long long stride_absmax;
    const float *diag; long long stride_diag;
    void *out; int out_dtype; long long stride_out;         // elements
};

// Launches of one chain on a stream (programmatic dependent launch): with `chained` the kernel may be brought onto the
// chip while its predecessor ends.  It calls chain_wait() before its first access to global memory - which returns when
// the predecessor is complete and its writes are visible, at once without the attribute - and chain_release() when its
// remaining work is short, so that a waiting successor does not hold SMs that other streams could use.
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool chained, A... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cfg.attrs = attr; cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

int launch_grad_planes(const void *stat_items, int n_stat, const void *split_items, int n_split, const long long *grads, float *part_amax,
                       float *part_ss, int *gexp, int target, void *plane_base, cudaStream_t stream);
int read_apply_error(bool clear);    // error words of the kernels in apply_kernels.cu and refresh.cu
int read_refresh_error(bool clear);
int launch_merge_t(const float *G, long long ldg, long long strideG, const float *Tp, long long strideTp, int wo, int count,
                   float *T, long long strideT, cudaStream_t stream, void *hi = nullptr, void *lo = nullptr, long long ldp = 0,
                   long long strideP = 0, int *exp_out = nullptr, int target = 0, bool chained = false);
int launch_quantize(const QuantArgs &a, cudaStream_t stream);
int launch_dequantize(const DequantArgs &a, cudaStream_t stream);
// a.out / a.out_dtype / a.stride_out are ignored: output goes to the bf16 planes hi, lo
// amax_scratch != nullptr: scaled fp16 planes (exponents from each matrix's largest magnitude and
// `target`, written to exp_out); nullptr: plain bf16 planes.
int launch_dequantize_planes(const DequantArgs &a, const int *slots, void *hi, void *lo, long long ldp, long long strideP,
                             cudaStream_t stream, float *amax_scratch = nullptr, int target = 0, int *exp_out = nullptr);
int launch_state_exponents(const float *absmax, long long stride_absmax, int n_absmax, const float *diag, long long stride_diag,
                           int n_diag, const int *slots, int count, int target, int *exp_out, cudaStream_t stream);
int launch_selftest_division(unsigned long long seed, unsigned long long pairs, unsigned long long *mismatches_dev,
                             cudaStream_t stream);
void set_panel_blocked(int on);
int launch_householder_panel(float *A, long long strideA, int n, int ld, int count, int j0, int w,
                             float *V, long long strideV, float *T, long long strideT, cudaStream_t stream,
                             int prev_w = 0, const float *Tprev = nullptr, int block_end = 0,
                             // scaled fp16 planes of V (see qr_kernels.cu); null: none
                             void *planes_hi = nullptr, void *planes_lo = nullptr, long long ldp = 0, long long strideP = 0,
                             int plane_col = 0, int rows_above = 0, int plane_exp = 0, bool chained = false);

}  // namespace qt
