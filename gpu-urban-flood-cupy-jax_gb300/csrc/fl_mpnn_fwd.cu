// The surrogate network's forward pass as fused blocks on the tensor cores:
//   k_edge_fwd  a processor layer's messages and their sum: for a tile of 128
//               receiving cells and each of their (at most three) incoming
//               edges, z1 = relu([h_i, h_j, e_ij] W1^T + b1), m = z1 W2^T + b2,
//               and agg_i = sum of the cell's messages in edge order
//   k_mlp2      a two-layer MLP over rows: the node update
//               h + W2 relu(W1 [h, agg] + b1) + b2, the encoders, the decoder
// One GEMM launch per product would write and read back every activation:
// per layer and cell 9.2 KB, of which 1.5 KB z1 and 3 KB fp32 messages; here
// z1 and the messages never leave the SM (z1 goes to the second product as a
// TMEM operand, the messages are summed in registers), 1.3 KB per layer and
// cell for the edge block and 1.8 KB for the node update.
//
// The edge block's tile rows are cells, not edges: edge slot k of the 128
// cells is one M = 128 product, so a cell's messages lie in one TMEM lane
// (and one thread) and their sum needs no exchange between threads, and the
// receiver's rows are staged once for the three slots.  A slot past a cell's
// last edge leaves its row stale; rows are independent and that one is not
// stored or summed.
//
// Measured (8 layers, 1.9 M cells and 5.7 M edges): 34.7 ms a pass with one
// launch per product, 12.0 ms here; per launch and 401,408 cells k_edge_fwd
// 156 us (the SM's shared-memory pipe 91 % busy: MMA operands, gathers, bias
// reads), k_mlp2 as node update 150 us (4.5 TB/s).
//
// Both kernels are persistent and warp-specialised like k_gemm_bf16_pers:
// four producer warps (cp.async gathers into 16 KB stages), one MMA lane,
// eight epilogue warps; weights stay in shared memory.  The rounding points
// (bf16 activations, fp32 accumulation in K order, fp32 sums in edge order)
// are those of the separate products, so both give the same bits.
//
// Every mbarrier wait is bounded; one that gives up sets the error flag.
#include "fl_mpnn.cuh"

namespace fl {

constexpr int MF_PROD_WARPS = 4, MF_EPI_WARPS = 8, MF_THREADS = 32 * (MF_PROD_WARPS + 1 + MF_EPI_WARPS);
constexpr int MF_CHUNKS = 14;  // 16 KB chunks of shared memory
constexpr int MF_SMEM = MF_CHUNKS * MM_CHUNK_BYTES + 1024 /* biases */ + 256 /* barriers */ + 1024 /* alignment */;
constexpr int EF_RING = 4;
constexpr int M2_MAX_RING = 8;

struct EdgeFwdArgs {
    const __nv_bfloat16 *h, *e;           // [C, 128], [E, 128]
    const int32_t *src, *start;           // [E], [C + 1]
    const __nv_bfloat16 *w1, *w2;         // [128, ldw1 >= 384], [128, ldw2 >= 128]
    int64_t ldw1, ldw2;
    const float *b1, *b2;
    __nv_bfloat16 *z1;                    // [E, 128] or nullptr
    __nv_bfloat16 *agg;                   // [C, 128]
    int32_t C;
    int32_t *error;
};

struct Mlp2Args {
    const __nv_bfloat16 *a[2];            // K segments
    int64_t lda[2];
    int32_t nk[2];                        // 64-wide chunks of each segment
    const __nv_bfloat16 *w1, *w2;         // [128, K], [n2, 128]
    int64_t ldw1, ldw2;
    const float *b1, *b2;
    const float *residual;                // [M, 128] or nullptr
    __nv_bfloat16 *z1;                    // [M, 128] or nullptr
    float *out_f32;                       // [M, n2] or nullptr
    __nv_bfloat16 *out_bf16;              // [M, n2] or nullptr
    int32_t n2, M, ring;
    int32_t *error;
};

// relu(v + bias) of 32 columns as 16 bf16 pairs; bias in shared memory.
__device__ __forceinline__ void relu_pack32(const uint32_t (&v)[32], const float *bias, uint32_t *out) {
#pragma unroll
    for (int q = 0; q < 32; q += 4) {
        const float4 b = *(const float4 *)(bias + q);
        out[q / 2] = pack_bf16x2(fmaxf(__uint_as_float(v[q]) + b.x, 0.0f), fmaxf(__uint_as_float(v[q + 1]) + b.y, 0.0f));
        out[q / 2 + 1] = pack_bf16x2(fmaxf(__uint_as_float(v[q + 2]) + b.z, 0.0f), fmaxf(__uint_as_float(v[q + 3]) + b.w, 0.0f));
    }
}

// One 128-deep second product: A = the z buffer in TMEM, B = w2 in shared memory.
__device__ __forceinline__ void mma_second(uint32_t d, uint32_t z, uint32_t sW2, uint32_t idesc) {
#pragma unroll
    for (int s = 0; s < MF_H / 16; ++s)
        umma_bf16_ts(d, z + 8u * s, umma_desc_sw128(sW2 + (s >> 2) * MM_CHUNK_BYTES + (s & 3) * 32), idesc, s > 0);
}

// TMEM: accumulator regions 0..2 (128 columns each), z buffers at 384 and 448.
__global__ void __launch_bounds__(MF_THREADS, 1) k_edge_fwd(const __grid_constant__ EdgeFwdArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sW1 = smem_addr(smem), sW2 = sW1 + 6 * MM_CHUNK_BYTES, sD = sW2 + 2 * MM_CHUNK_BYTES;
    const uint32_t sR = sD + 2 * MM_CHUNK_BYTES;
    float *bias = (float *)(smem + MF_CHUNKS * MM_CHUNK_BYTES);  // b1, b2
    uint64_t *bars = (uint64_t *)(bias + 256);
    const uint32_t dstf = smem_addr(bars), dste = dstf + 8, ringf = dstf + 16, ringe = ringf + 8 * EF_RING;
    const uint32_t d1f = ringe + 8 * EF_RING, zf = d1f + 24, d2f = zf + 16, de = d2f + 24, drain = de + 24;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 + 2 * EF_RING + 3 + 2 + 3 + 3 + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = (g.C + MM_BM - 1) / MM_BM;

    if (tid == 0) {
        mbar_init(dstf, 32 * MF_PROD_WARPS);
        mbar_init(dste, 1);
        for (int s = 0; s < EF_RING; ++s) {
            mbar_init(ringf + 8 * s, 32 * MF_PROD_WARPS);
            mbar_init(ringe + 8 * s, 1);
        }
        for (int k = 0; k < 3; ++k) {
            mbar_init(d1f + 8 * k, 1);
            mbar_init(d2f + 8 * k, 1);
            mbar_init(de + 8 * k, MF_EPI_WARPS);
        }
        mbar_init(zf, MF_EPI_WARPS);
        mbar_init(zf + 8, MF_EPI_WARPS);
        mbar_init(drain, 1);
        mbar_fence_init();
    }
    if (warp == MF_PROD_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // weights: not written by the kernel before this one (they change between passes only)
    for (int c = 0; c < 6; ++c) load_weight_chunk(g.w1, g.ldw1, MF_H, c, sW1 + c * MM_CHUNK_BYTES, tid, MF_THREADS);
    for (int c = 0; c < 2; ++c) load_weight_chunk(g.w2, g.ldw2, MF_H, c, sW2 + c * MM_CHUNK_BYTES, tid, MF_THREADS);
    if (tid < 256) bias[tid] = tid < 128 ? g.b1[tid] : g.b2[tid - 128];
    cp_async_commit();
    cp_async_wait_all();
    fence_async_smem();
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool bad = false;
    pdl_wait();  // the previous kernel's activations; only then may the next one start
    pdl_launch_dependents();

    if (warp < MF_PROD_WARPS) {
        // producers: lane = tile row 32 * warp + lane
        int t = blockIdx.x;
        int c = t * MM_BM + 32 * warp + lane;
        int rs = 0, re = 0, s0 = 0, s1 = 0, s2 = 0;
        if (t < tiles && c < g.C) {
            rs = g.start[c];
            re = g.start[c + 1];
            if (rs < re) s0 = g.src[rs];
            if (rs + 1 < re) s1 = g.src[rs + 1];
            if (rs + 2 < re) s2 = g.src[rs + 2];
        }
        int q = 0;
        for (int i = 0; t < tiles && !bad; ++i) {
            // the next tile's index loads are issued here and used in the next round
            const int tn = t + gridDim.x, cn = tn * MM_BM + 32 * warp + lane;
            int rsn = 0, ren = 0, n0 = 0, n1 = 0, n2 = 0;
            const bool more = tn < tiles && cn < g.C;
            if (more) {
                rsn = g.start[cn];
                ren = g.start[cn + 1];
            }
            if (i > 0 && !warp_wait(dste, (i - 1) & 1)) {
                bad = true;
                break;
            }
            const __nv_bfloat16 *own = c < g.C ? g.h + (int64_t)c * MF_H : nullptr;
            warp_copy_rows(own, sD, warp, lane);
            warp_copy_rows(own ? own + 64 : nullptr, sD + MM_CHUNK_BYTES, warp, lane);
            cp_async_arrive_noinc(dstf);
            if (more) {
                if (rsn < ren) n0 = g.src[rsn];
                if (rsn + 1 < ren) n1 = g.src[rsn + 1];
                if (rsn + 2 < ren) n2 = g.src[rsn + 2];
            }
#pragma unroll 1
            for (int k = 0; k < 3 && !bad; ++k) {
                const bool valid = rs + k < re;
                const int sk = k == 0 ? s0 : (k == 1 ? s1 : s2);
                const __nv_bfloat16 *ph = valid ? g.h + (int64_t)sk * MF_H : nullptr;
                const __nv_bfloat16 *pe = valid ? g.e + (int64_t)(rs + k) * MF_H : nullptr;
#pragma unroll
                for (int j = 0; j < 4; ++j, ++q) {
                    const int s = q % EF_RING, u = q / EF_RING;
                    if (u > 0 && !warp_wait(ringe + 8 * s, (u - 1) & 1)) {
                        bad = true;
                        break;
                    }
                    const __nv_bfloat16 *p = j < 2 ? ph : pe;
                    warp_copy_rows(p ? p + (j & 1) * 64 : nullptr, sR + s * MM_CHUNK_BYTES, warp, lane);
                    cp_async_arrive_noinc(ringf + 8 * s);
                }
            }
            t = tn; c = cn; rs = rsn; re = ren; s0 = n0; s1 = n1; s2 = n2;
        }
        cp_async_wait_all();
    } else if (warp == MF_PROD_WARPS) {
        // the whole warp runs the loop, so its control and descriptors stay in
        // uniform registers; one elected lane issues
        const bool issuer = elect_one();
        {
            // slot n = 3 i + k: its first product goes to region k, then the
            // second product of slot n - 1 (whose z the epilogue wrote meanwhile)
            const uint32_t idesc = umma_idesc_bf16_128x128();
            int q = 0, i = 0, n = 0;
            auto second = [&](int m, int k) {
                if (!warp_wait(zf + 8 * (m & 1), (m >> 1) & 1)) {
                    bad = true;
                    return;
                }
                tmem_fence_after();
                if (issuer) {
                    mma_second(tmem + (uint32_t)(k * 128), tmem + 384u + 64u * (m & 1), sW2, idesc);
                    umma_commit(d2f + 8 * k);
                }
            };
            for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x, ++i) {
                if (!warp_wait(dstf, i & 1)) {
                    bad = true;
                    break;
                }
                fence_async_smem();
#pragma unroll 1
                for (int k = 0; k < 3 && !bad; ++k, ++n) {
                    if (i > 0 && !warp_wait(de + 8 * k, (i - 1) & 1)) {
                        bad = true;
                        break;
                    }
                    tmem_fence_after();
                    const uint32_t d = tmem + (uint32_t)(k * 128);
                    if (issuer) {
#pragma unroll
                        for (int s = 0; s < 8; ++s)
                            umma_bf16(d, umma_desc_sw128(sD + (s >> 2) * MM_CHUNK_BYTES + (s & 3) * 32),
                                      umma_desc_sw128(sW1 + (s >> 2) * MM_CHUNK_BYTES + (s & 3) * 32), idesc, s > 0);
                        if (k == 2) umma_commit(dste);
                    }
                    for (int j = 0; j < 4; ++j, ++q) {
                        const int st = q % EF_RING;
                        if (!warp_wait(ringf + 8 * st, (q / EF_RING) & 1)) {
                            bad = true;
                            break;
                        }
                        fence_async_smem();
                        const uint32_t a0 = sR + st * MM_CHUNK_BYTES, b0 = sW1 + (2 + j) * MM_CHUNK_BYTES;
                        if (issuer) {
#pragma unroll
                            for (int s = 0; s < 4; ++s)
                                umma_bf16(d, umma_desc_sw128(a0 + s * 32), umma_desc_sw128(b0 + s * 32), idesc, 1u);
                            umma_commit(ringe + 8 * st);
                        }
                    }
                    if (bad) break;
                    if (issuer) umma_commit(d1f + 8 * k);
                    if (n > 0) second(n - 1, k == 0 ? 2 : k - 1);
                }
            }
            if (n > 0 && !bad) second(n - 1, 2);
            // every MMA issued so far has completed before TMEM is released
            if (issuer) umma_commit(drain);
            (void)warp_wait(drain, 0);
        }
    } else {
        // epilogue: thread = one cell, 64 of its 128 columns
        const int quad = warp & 3, half = (warp - MF_PROD_WARPS - 1) >> 2;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        const float *b1 = bias + half * 64, *b2 = bias + 128 + half * 64;
        float acc[64];
        int n = 0, pc = 0, pdeg = 0;
        // the messages of slot m (region k) of cell cc: summed, and stored after the last
        auto sum_slot = [&](int m, int k, int cc, int deg) {
            if (!warp_wait(d2f + 8 * k, (m / 3) & 1)) {
                bad = true;
                return;
            }
            tmem_fence_after();
            const bool valid = k < deg;
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                uint32_t v[32];
                tmem_ld32(tmem + lanes + (uint32_t)(k * 128 + half * 64 + hh * 32), v);
                if (hh == 1) {
                    tmem_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(de + 8 * k);
                }
#pragma unroll
                for (int u = 0; u < 32; u += 4) {
                    const float4 b = *(const float4 *)(b2 + hh * 32 + u);
                    const float x[4] = {__uint_as_float(v[u]) + b.x, __uint_as_float(v[u + 1]) + b.y,
                                        __uint_as_float(v[u + 2]) + b.z, __uint_as_float(v[u + 3]) + b.w};
#pragma unroll
                    for (int w = 0; w < 4; ++w) {
                        const float a = k == 0 ? 0.0f : acc[hh * 32 + u + w];
                        acc[hh * 32 + u + w] = valid ? a + x[w] : a;
                    }
                }
            }
            if (k == 2 && cc < g.C) {
                __nv_bfloat16 *p = g.agg + (int64_t)cc * MF_H + half * 64;
#pragma unroll
                for (int u = 0; u < 64; u += 16) {
                    uint32_t w[8];
#pragma unroll
                    for (int x = 0; x < 8; ++x) w[x] = pack_bf16x2(acc[u + 2 * x], acc[u + 2 * x + 1]);
                    st8u(p + u, w);
                }
            }
            __syncwarp();
        };
        for (int t = blockIdx.x, i = 0; t < tiles && !bad; t += gridDim.x, ++i) {
            const int c = t * MM_BM + quad * 32 + lane;
            int rs = 0, deg = 0;
            if (c < g.C) {
                rs = g.start[c];
                deg = g.start[c + 1] - rs;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k, ++n) {
                if (!warp_wait(d1f + 8 * k, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
                const uint32_t z = tmem + lanes + 384u + 64u * (n & 1) + (uint32_t)(half * 32);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t v[32], w[16];
                    tmem_ld32(tmem + lanes + (uint32_t)(k * 128 + half * 64 + hh * 32), v);
                    relu_pack32(v, b1 + hh * 32, w);
                    tmem_st16(z + (uint32_t)(hh * 16), w);
                    if (g.z1 && k < deg) {
                        __nv_bfloat16 *p = g.z1 + (int64_t)(rs + k) * MF_H + half * 64 + hh * 32;
                        st8u(p, w);
                        st8u(p + 16, w + 8);
                    }
                    __syncwarp();
                }
                tmem_wait_st();
                tmem_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(zf + 8 * (n & 1));
                if (n > 0) sum_slot(n - 1, k == 0 ? 2 : k - 1, k == 0 ? pc : c, k == 0 ? pdeg : deg);
                if (bad) break;
            }
            pc = c;
            pdeg = deg;
        }
        if (n > 0 && !bad) sum_slot(n - 1, 2, pc, pdeg);
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    tmem_fence_before();
    __syncthreads();
    if (warp == MF_PROD_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

__global__ void __launch_bounds__(MF_THREADS, 1) k_mlp2(const __grid_constant__ Mlp2Args g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int nK = g.nk[0] + g.nk[1], S = g.ring;
    const uint32_t sW1 = smem_addr(smem), sW2 = sW1 + nK * MM_CHUNK_BYTES, sR = sW2 + 2 * MM_CHUNK_BYTES;
    float *bias = (float *)(smem + MF_CHUNKS * MM_CHUNK_BYTES);
    uint64_t *bars = (uint64_t *)(bias + 256);
    const uint32_t ringf = smem_addr(bars), ringe = ringf + 8 * M2_MAX_RING;
    const uint32_t d1f = ringe + 8 * M2_MAX_RING, zf = d1f + 24, d2f = zf + 16, de = d2f + 24, drain = de + 24;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * M2_MAX_RING + 3 + 2 + 3 + 3 + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = (g.M + MM_BM - 1) / MM_BM;

    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(ringf + 8 * s, 32 * MF_PROD_WARPS);
            mbar_init(ringe + 8 * s, 1);
        }
        for (int k = 0; k < 3; ++k) {
            mbar_init(d1f + 8 * k, 1);
            mbar_init(d2f + 8 * k, 1);
            mbar_init(de + 8 * k, MF_EPI_WARPS);
        }
        mbar_init(zf, MF_EPI_WARPS);
        mbar_init(zf + 8, MF_EPI_WARPS);
        mbar_init(drain, 1);
        mbar_fence_init();
    }
    if (warp == MF_PROD_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    for (int c = 0; c < nK; ++c) load_weight_chunk(g.w1, g.ldw1, MF_H, c, sW1 + c * MM_CHUNK_BYTES, tid, MF_THREADS);
    for (int c = 0; c < 2; ++c) load_weight_chunk(g.w2, g.ldw2, g.n2, c, sW2 + c * MM_CHUNK_BYTES, tid, MF_THREADS);
    if (tid < 256) bias[tid] = tid < 128 ? g.b1[tid] : (tid - 128 < g.n2 ? g.b2[tid - 128] : 0.0f);
    cp_async_commit();
    cp_async_wait_all();
    fence_async_smem();
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool bad = false;
    pdl_wait();
    pdl_launch_dependents();

    if (warp < MF_PROD_WARPS) {
        int q = 0;
        for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x) {
            const int r = t * MM_BM + 32 * warp + lane;
            const __nv_bfloat16 *p0 = r < g.M ? g.a[0] + (int64_t)r * g.lda[0] : nullptr;
            const __nv_bfloat16 *p1 = r < g.M && g.nk[1] ? g.a[1] + (int64_t)r * g.lda[1] : nullptr;
            for (int c = 0; c < nK; ++c, ++q) {
                const int s = q % S, u = q / S;
                if (u > 0 && !warp_wait(ringe + 8 * s, (u - 1) & 1)) {
                    bad = true;
                    break;
                }
                const __nv_bfloat16 *p = c < g.nk[0] ? p0 : p1;
                const int col = (c < g.nk[0] ? c : c - g.nk[0]) * 64;
                warp_copy_rows(p ? p + col : nullptr, sR + s * MM_CHUNK_BYTES, warp, lane);
                cp_async_arrive_noinc(ringf + 8 * s);
            }
        }
        cp_async_wait_all();
    } else if (warp == MF_PROD_WARPS) {
        // the whole warp runs the loop, so its control and descriptors stay in
        // uniform registers; one elected lane issues
        const bool issuer = elect_one();
        {
            const uint32_t idesc = umma_idesc_bf16_128x128();
            int q = 0, n = 0;
            auto second = [&](int m) {
                const int k = m % 3;
                if (!warp_wait(zf + 8 * (m & 1), (m >> 1) & 1)) {
                    bad = true;
                    return;
                }
                tmem_fence_after();
                if (issuer) {
                    mma_second(tmem + (uint32_t)(k * 128), tmem + 384u + 64u * (m & 1), sW2, idesc);
                    umma_commit(d2f + 8 * k);
                }
            };
            for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x, ++n) {
                const int k = n % 3;
                if (n >= 3 && !warp_wait(de + 8 * k, (n / 3 - 1) & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
                const uint32_t d = tmem + (uint32_t)(k * 128);
                for (int c = 0; c < nK; ++c, ++q) {
                    const int st = q % S;
                    if (!warp_wait(ringf + 8 * st, (q / S) & 1)) {
                        bad = true;
                        break;
                    }
                    fence_async_smem();
                    const uint32_t a0 = sR + st * MM_CHUNK_BYTES, b0 = sW1 + c * MM_CHUNK_BYTES;
                    if (issuer) {
#pragma unroll
                        for (int s = 0; s < 4; ++s)
                            umma_bf16(d, umma_desc_sw128(a0 + s * 32), umma_desc_sw128(b0 + s * 32), idesc,
                                      (c > 0 || s > 0) ? 1u : 0u);
                        umma_commit(ringe + 8 * st);
                    }
                }
                if (bad) break;
                if (issuer) umma_commit(d1f + 8 * k);
                if (n > 0) second(n - 1);
            }
            if (n > 0 && !bad) second(n - 1);
            if (issuer) umma_commit(drain);
            (void)warp_wait(drain, 0);
        }
    } else {
        const int quad = warp & 3, half = (warp - MF_PROD_WARPS - 1) >> 2;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        const float *b1 = bias + half * 64, *b2 = bias + 128 + half * 64;
        const bool has_out = half * 64 < g.n2;  // (n2 = 64: the upper columns do not exist)
        int n = 0, pr = 0;
        auto finish = [&](int m, int r) {
            const int k = m % 3;
            float res[32];
            const float *rp = g.residual && r < g.M ? g.residual + (int64_t)r * MF_H + half * 64 : nullptr;
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                if (rp) {
#pragma unroll
                    for (int u = 0; u < 32; u += 8) ld8f(rp + hh * 32 + u, res + u);
                }
                if (hh == 0) {
                    if (!warp_wait(d2f + 8 * k, (m / 3) & 1)) {
                        bad = true;
                        return;
                    }
                    tmem_fence_after();
                }
                uint32_t v[32];
                tmem_ld32(tmem + lanes + (uint32_t)(k * 128 + half * 64 + hh * 32), v);
                if (hh == 1) {
                    tmem_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(de + 8 * k);
                }
                if (has_out && r < g.M) {
                    float x[32];
#pragma unroll
                    for (int u = 0; u < 32; u += 4) {
                        const float4 b = *(const float4 *)(b2 + hh * 32 + u);
                        x[u] = __uint_as_float(v[u]) + b.x;
                        x[u + 1] = __uint_as_float(v[u + 1]) + b.y;
                        x[u + 2] = __uint_as_float(v[u + 2]) + b.z;
                        x[u + 3] = __uint_as_float(v[u + 3]) + b.w;
                    }
                    if (rp) {
#pragma unroll
                        for (int u = 0; u < 32; ++u) x[u] += res[u];
                    }
                    const int64_t o = (int64_t)r * g.n2 + half * 64 + hh * 32;
                    if (g.out_f32) {
#pragma unroll
                        for (int u = 0; u < 32; u += 8) st8f(g.out_f32 + o + u, x + u);
                    }
                    if (g.out_bf16) {
#pragma unroll
                        for (int u = 0; u < 32; u += 16) {
                            uint32_t w[8];
#pragma unroll
                            for (int y = 0; y < 8; ++y) w[y] = pack_bf16x2(x[u + 2 * y], x[u + 2 * y + 1]);
                            st8u(g.out_bf16 + o + u, w);
                        }
                    }
                }
                __syncwarp();
            }
        };
        for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x, ++n) {
            const int r = t * MM_BM + quad * 32 + lane, k = n % 3;
            if (!warp_wait(d1f + 8 * k, (n / 3) & 1)) {
                bad = true;
                break;
            }
            tmem_fence_after();
            const uint32_t z = tmem + lanes + 384u + 64u * (n & 1) + (uint32_t)(half * 32);
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                uint32_t v[32], w[16];
                tmem_ld32(tmem + lanes + (uint32_t)(k * 128 + half * 64 + hh * 32), v);
                relu_pack32(v, b1 + hh * 32, w);
                tmem_st16(z + (uint32_t)(hh * 16), w);
                if (g.z1 && r < g.M) {
                    __nv_bfloat16 *p = g.z1 + (int64_t)r * MF_H + half * 64 + hh * 32;
                    st8u(p, w);
                    st8u(p + 16, w + 8);
                }
                __syncwarp();
            }
            tmem_wait_st();
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(zf + 8 * (n & 1));
            if (n > 0) finish(n - 1, pr);
            pr = r;
        }
        if (n > 0 && !bad) finish(n - 1, pr);
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    tmem_fence_before();
    __syncthreads();
    if (warp == MF_PROD_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

}  // namespace fl

using namespace fl;

extern "C" FL_API int fl_mpnn_forward(const FlMpnnForwardDesc *d, void *stream) {
    if (!d || d->cells < 1 || d->edges < 0 || d->layers < 0) return set_error(FL_E_INVALID, "fl_mpnn_forward: bad sizes");
    const bool edges = d->edges > 0;
    if (!d->x || !d->y || !d->recv_start || !d->h_f32[0] || !d->h_f32[1] || !d->h_bf || (edges && (!d->src || !d->ef || !d->e)) ||
        (d->layers > 0 && (!d->edge || !d->node || !d->agg)))
        return set_error(FL_E_INVALID, "fl_mpnn_forward: NULL pointer");
    if (d->ldx < 64 || d->ldx % 8 || d->lde < 64 || d->lde % 8)
        return set_error(FL_E_INVALID, "fl_mpnn_forward: leading dimensions must be multiples of 8 and at least 64");
    uintptr_t a16 = (uintptr_t)d->x | (uintptr_t)d->ef;
    uintptr_t a32 = (uintptr_t)d->y | (uintptr_t)d->h_f32[0] | (uintptr_t)d->h_f32[1] | (uintptr_t)d->zn | (uintptr_t)d->ze |
                    (uintptr_t)d->e | (uintptr_t)d->zd;
    auto dense = [&](const FlDenseRef &r, int k) {
        a16 |= (uintptr_t)r.w;
        return r.w && r.b && r.ldw >= k && r.ldw % 8 == 0;
    };
    bool ok = dense(d->enc_n[0], 64) && dense(d->enc_n[1], 128) && dense(d->enc_e[0], 64) && dense(d->enc_e[1], 128) &&
              dense(d->dec[0], 128) && dense(d->dec[1], 128);
    for (int l = 0; l < d->layers; ++l) {
        ok = ok && dense(d->edge[2 * l], 384) && dense(d->edge[2 * l + 1], 128) && dense(d->node[2 * l], 256) &&
             dense(d->node[2 * l + 1], 128) && d->agg[l] && d->h_bf[l];
        if (!ok) break;
        a32 |= (uintptr_t)d->agg[l] | (uintptr_t)d->h_bf[l] | (uintptr_t)(d->z1e ? d->z1e[l] : nullptr) |
               (uintptr_t)(d->z1n ? d->z1n[l] : nullptr);
    }
    if (!ok || !d->h_bf[d->layers]) return set_error(FL_E_INVALID, "fl_mpnn_forward: bad layer");
    a32 |= (uintptr_t)d->h_bf[d->layers];
    if (a16 % 16 || a32 % 32)
        return set_error(FL_E_INVALID, "fl_mpnn_forward: inputs and weights must be 16-byte, buffers 32-byte aligned");
    int32_t *err = nullptr;
    int rc = gemm_error_flag(&err);
    if (rc) return rc;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    static std::atomic<uint64_t> edge_done{0}, mlp_done{0};
    if (e == cudaSuccess) e = allow_smem((const void *)k_edge_fwd, MF_SMEM, dev, edge_done);
    if (e == cudaSuccess) e = allow_smem((const void *)k_mlp2, MF_SMEM, dev, mlp_done);
    cudaStream_t st = (cudaStream_t)stream;
    using bf = __nv_bfloat16;
    int64_t launched = 0;
    auto mlp = [&](const void *a0, int64_t ld0, int k0, const void *a1, int k1, const FlDenseRef &w1, const FlDenseRef &w2,
                   int n2, int rows, const float *res, void *z, float *of, void *ob) {
        if (e != cudaSuccess) return;
        Mlp2Args m{};
        m.a[0] = (const bf *)a0;
        m.a[1] = (const bf *)a1;
        m.lda[0] = ld0;
        m.lda[1] = MF_H;
        m.nk[0] = k0 / 64;
        m.nk[1] = k1 / 64;
        m.w1 = (const bf *)w1.w;
        m.ldw1 = w1.ldw;
        m.b1 = w1.b;
        m.w2 = (const bf *)w2.w;
        m.ldw2 = w2.ldw;
        m.b2 = w2.b;
        m.residual = res;
        m.z1 = (bf *)z;
        m.out_f32 = of;
        m.out_bf16 = (bf *)ob;
        m.n2 = n2;
        m.M = rows;
        m.ring = std::min(M2_MAX_RING, MF_CHUNKS - 2 - (k0 + k1) / 64);
        m.error = err;
        e = launch_blocks(k_mlp2, m, (rows + MM_BM - 1) / MM_BM, sms, MF_THREADS, MF_SMEM, launched > 0, st);
        ++launched;
    };
    mlp(d->x, d->ldx, 64, nullptr, 0, d->enc_n[0], d->enc_n[1], MF_H, d->cells, nullptr, d->zn, d->h_f32[0], d->h_bf[0]);
    if (edges) mlp(d->ef, d->lde, 64, nullptr, 0, d->enc_e[0], d->enc_e[1], MF_H, d->edges, nullptr, d->ze, nullptr, d->e);
    for (int l = 0; l < d->layers && e == cudaSuccess; ++l) {
        EdgeFwdArgs q{};
        q.h = (const bf *)d->h_bf[l];
        q.e = (const bf *)d->e;
        q.src = d->src;
        q.start = d->recv_start;
        q.w1 = (const bf *)d->edge[2 * l].w;
        q.ldw1 = d->edge[2 * l].ldw;
        q.b1 = d->edge[2 * l].b;
        q.w2 = (const bf *)d->edge[2 * l + 1].w;
        q.ldw2 = d->edge[2 * l + 1].ldw;
        q.b2 = d->edge[2 * l + 1].b;
        q.z1 = d->z1e ? (bf *)d->z1e[l] : nullptr;
        q.agg = (bf *)d->agg[l];
        q.C = d->cells;
        q.error = err;
        e = launch_blocks(k_edge_fwd, q, (d->cells + MM_BM - 1) / MM_BM, sms, MF_THREADS, MF_SMEM, true, st);
        ++launched;
        mlp(d->h_bf[l], MF_H, 128, d->agg[l], 128, d->node[2 * l], d->node[2 * l + 1], MF_H, d->cells, d->h_f32[l & 1],
            d->z1n ? d->z1n[l] : nullptr, d->h_f32[(l & 1) ^ 1], d->h_bf[l + 1]);
    }
    mlp(d->h_bf[d->layers], MF_H, 128, nullptr, 0, d->dec[0], d->dec[1], 64, d->cells, nullptr, d->zd, d->y, nullptr);
    if (e != cudaSuccess) return set_error(FL_E_CUDA, "fl_mpnn_forward: %s", cudaGetErrorString(e));
    add_launches(launched);
    return FL_OK;
}
