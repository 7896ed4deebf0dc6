// tcgen05 / TMEM helpers shared by the tensor-core kernels (fl_mlp.cu, fl_mpnn_fwd.cu,
// fl_mpnn_bwd.cu): shared-memory and instruction descriptors, MMA issue with A in
// shared memory or in TMEM, TMEM loads and stores, 32-byte global accesses.
#pragma once

#include <cuda_bf16.h>

#include "fl_device.cuh"

namespace fl {

constexpr int MM_BM = 128, MM_BN = 128, MM_BK = 64;
constexpr int MM_CHUNK_BYTES = MM_BM * MM_BK * 2;  // 16 KB per operand per stage
constexpr uint64_t MM_WAIT_NS = 1000000000ull;

__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);  // start address (16-byte units)
    d |= (uint64_t)1 << 16;                    // leading byte offset (unused by swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1 << 46;                    // descriptor version
    d |= (uint64_t)2 << 61;                    // 128-byte swizzle
    return d;
}

// Operand stored with its M (N) index contiguous, 128-byte swizzle: 64 of them
// (128 bytes) per K row, 8-row groups 1024 bytes apart, the next 64 of them
// `block` bytes on.
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t saddr, uint32_t block) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(block >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Instruction descriptor with both operands M (N) contiguous, M = 128, N = n.
__device__ __forceinline__ uint32_t umma_idesc_bf16_mn(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(MM_BM >> 4) << 24);
}

// kind::f16 instruction descriptor: fp32 accumulator, bf16 A and B, both
// K-major, M = 128, N = 128.
__device__ __forceinline__ uint32_t umma_idesc_bf16_128x128() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MM_BN >> 3) << 17) | ((uint32_t)(MM_BM >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.u32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

// One lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n"
        ".reg .pred q;\n"
        "elect.sync _|q, 0xffffffff;\n"
        "selp.u32 %0, 1, 0, q;\n"
        "}\n"
        : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 32-byte global accesses (8 x 32 bits; the address is 32-byte aligned).
__device__ __forceinline__ void ld8f(const float *p, float *d) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]), "=f"(d[4]), "=f"(d[5]), "=f"(d[6]), "=f"(d[7])
                 : "l"(p));
}
__device__ __forceinline__ void st8f(float *p, const float *s) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(s[0]), "f"(s[1]), "f"(s[2]),
                 "f"(s[3]), "f"(s[4]), "f"(s[5]), "f"(s[6]), "f"(s[7])
                 : "memory");
}
__device__ __forceinline__ void st8u(void *p, const uint32_t *s) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(s[0]), "r"(s[1]), "r"(s[2]),
                 "r"(s[3]), "r"(s[4]), "r"(s[5]), "r"(s[6]), "r"(s[7])
                 : "memory");
}

// A in TMEM (row = lane; 16 K values of a step in 8 columns, two per column), B in shared memory.
__device__ __forceinline__ void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.u32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The mma-fragment shapes: 16 lanes (rows) from taddr's, 32 columns.  Lane
// l = 4 g + q of the warp holds rows g and g + 8; of each 8-column block j the
// columns 8 j + 2 q and + 1: r[4 j + 0, 1] of row g, r[4 j + 2, 3] of row g + 8.
__device__ __forceinline__ void tmem_ld_frag32(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The same columns as packed pairs (16 words a row): r[2 j] of row g, r[2 j + 1] of row g + 8.
__device__ __forceinline__ void tmem_st_frag_pairs(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

// 4 x 4 transpose over the lanes q = 0..3 of a group of four: afterwards word p
// of lane q is what word q of lane p was.
__device__ __forceinline__ void transpose4(uint32_t &w0, uint32_t &w1, uint32_t &w2, uint32_t &w3, int q) {
    const bool o1 = (q & 1) != 0, o2 = (q & 2) != 0;
    uint32_t a = __shfl_xor_sync(0xffffffffu, o1 ? w0 : w1, 1), b = __shfl_xor_sync(0xffffffffu, o1 ? w2 : w3, 1);
    if (o1) {
        w0 = a;
        w2 = b;
    } else {
        w1 = a;
        w3 = b;
    }
    a = __shfl_xor_sync(0xffffffffu, o2 ? w0 : w2, 2);
    b = __shfl_xor_sync(0xffffffffu, o2 ? w1 : w3, 2);
    if (o2) {
        w0 = a;
        w1 = b;
    } else {
        w2 = a;
        w3 = b;
    }
}

__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// A bounded wait of a whole warp: one outcome for all lanes, which then go on
// together (the TMEM accesses that follow are warp-wide).
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, MM_WAIT_NS));
}

// 32 rows of a 128-row chunk (those from 32 pw), by one warp: four whole 128-byte
// row pieces per instruction.  Lane l copies the rows 4 i + l / 8, whose numbers
// it holds itself (row[i]; < 0: the row is left as it is), from `base`, the
// matrix at the chunk's first column.  The numbers are exchanged once for all
// chunks of a row (rows_of_lane): a shuffled pointer per copy instruction took
// two of every six cycles of the pipe that also writes the copies.
__device__ __forceinline__ void warp_copy_numbered(const __nv_bfloat16 *base, int64_t ld, const int (&row)[8], uint32_t sdst, int pw,
                                                   int lane) {
    const int c = lane & 7;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int R = 32 * pw + 4 * i + (lane >> 3);
        if (row[i] >= 0) cp_async16(sdst + (uint32_t)(R * 128 + ((c ^ (R & 7)) << 4)), base + row[i] * ld + c * 8);
    }
}

// ROWS consecutive rows of a matrix from `first` (those past `limit` are left
// as they are) to the rows R0 .. of a chunk.
template <int ROWS>
__device__ __forceinline__ void warp_copy_span(const __nv_bfloat16 *base, int64_t ld, int64_t first, int64_t limit, uint32_t sdst,
                                               int R0, int lane) {
    const int c = lane & 7;
#pragma unroll
    for (int i = 0; i < ROWS / 4; ++i) {
        const int rr = 4 * i + (lane >> 3), R = R0 + rr;
        if (first + rr < limit) cp_async16(sdst + (uint32_t)(R * 128 + ((c ^ (R & 7)) << 4)), base + (first + rr) * ld + c * 8);
    }
}

// own: a value per tile row of the warp (lane = row) to the lanes that copy them.
__device__ __forceinline__ void rows_of_lane(int own, int (&row)[8], int lane) {
#pragma unroll
    for (int i = 0; i < 8; ++i) row[i] = __shfl_sync(0xffffffffu, own, 4 * i + (lane >> 3));
}

// 64-wide K chunk c of a bf16 matrix's rows [0, n) into the K-major 128-byte-swizzle layout at
// sdst (rows n .. 127 zeroed); every thread of the block takes part, cp.async.
__device__ __forceinline__ void load_weight_chunk(const __nv_bfloat16 *w, int64_t ldw, int n, int c, uint32_t sdst,
                                                  int tid, int threads) {
    for (int p = tid; p < MM_BN * 8; p += threads) {
        const int R = p >> 3, cc = p & 7;
        const uint32_t dst = sdst + (uint32_t)(R * 128 + ((cc ^ (R & 7)) << 4));
        if (R < n) cp_async16(dst, w + (int64_t)R * ldw + c * MM_BK + cc * 8);
        else asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "r"(0u) : "memory");
    }
}

__device__ __forceinline__ void ld8u(const void *p, uint32_t *d) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7])
                 : "l"(p));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *(uint32_t *)&h;
}

}  // namespace fl
