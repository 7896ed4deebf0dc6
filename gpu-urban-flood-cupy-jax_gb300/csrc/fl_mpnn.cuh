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

// Producer warp's part of a 128-row chunk: its 32 rows, four whole 128-byte
// row pieces per instruction.  `own`: this lane's row pointer (nullptr: the
// row is left as it is), at the chunk's first column.
__device__ __forceinline__ void warp_copy_rows(const __nv_bfloat16 *own, uint32_t sdst, int pw, int lane) {
    const int c = lane & 7;
    const uint64_t p = (uint64_t)own;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int rr = 4 * i + (lane >> 3);
        const uint64_t row = __shfl_sync(0xffffffffu, p, rr);
        const int R = 32 * pw + rr;
        if (row) cp_async16(sdst + (uint32_t)(R * 128 + ((c ^ (R & 7)) << 4)), (const __nv_bfloat16 *)row + c * 8);
    }
}

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
