// Shared by the surrogate network's forward and backward blocks (fl_mpnn_fwd.cu, fl_mpnn_bwd.cu).
#pragma once

#include <algorithm>
#include <atomic>

#include "fl_umma.cuh"

namespace fl {

int set_error(int code, const char *fmt, ...);
void add_launches(int64_t n);
int gemm_error_flag(int32_t **out);

constexpr int MF_H = 128;  // hidden width

// Raise a kernel's dynamic shared memory limit once per device.
inline cudaError_t allow_smem(const void *fn, int bytes, int dev, std::atomic<uint64_t> &done) {
    if (dev < 64 && (done.load(std::memory_order_acquire) >> dev & 1u)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev < 64) done.fetch_or(1ull << dev, std::memory_order_release);
    return e;
}

// A pass's launches after the first are programmatic dependents of the one
// before: a block's set-up (TMEM, weights) overlaps the previous kernel's
// last tiles.  A kernel lets its dependent start only after its own wait, so
// a prefetch of weights never overtakes a kernel before the pass.
template <class Args>
inline cudaError_t launch_blocks(void (*kernel)(Args), const Args &a, int blocks, int sms, int threads, int smem,
                                 bool dependent, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::max(1, std::min(blocks, sms)));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

}  // namespace fl
