// The surrogate network's backward pass as fused blocks on the tensor cores:
//   k_mlp_bwd    a two-layer MLP's backward over rows: dz2 = bf16(dy), dz1 =
//                relu'(z) (dz2 W2), dx = dz1 W1, with the bias gradients
//                (column sums of the fp32 values) on the way; for a processor
//                layer also dh = dy + dx, the message gradient
//                dagg = dz1 W1[:, 128:], and per incoming edge of a cell
//                dz_e = relu'(z1_e) (dagg W_e2) -- one product per cell, as
//                all of a cell's messages have the same gradient
//   k_edge_bwd   dh += sum over the cell's incoming edges of dz_e W_e1[dst] +
//                sum over its outgoing edges of dz_e W_e1[src]: gathers the
//                128-wide dz_e rows instead of writing 384-wide fp32 input
//                gradients and gathering those
//   k_edge_dsum  the edge encoder's output gradient sum_l dz_e(l) W_e1(l)[e]
//                over all layers' dz_e at the end, instead of a fp32 [E, 128]
//                running sum read and written by every layer
//   k_wgrad      the weight gradients dZ^T X of a layer's products in one
//                launch: rows are the reduction index, so both operands are
//                read as they lie in memory (M / N contiguous descriptors);
//                no transposed copies.  Each CTA reduces a fixed range of rows
//   k_reduce     the CTAs' partial sums, in CTA order, into the gradients
// Activation gradients keep the rounding points and orders of sums of the
// separate products (same bits); weight and bias gradients are fp32 sums over
// rows in a fixed order.
//
// Measured: one optimizer step on 100,352 cells and 299,712 dual edges, 8
// layers: see the figures at fl_mpnn_backward.
//
// Every mbarrier wait is bounded; one that gives up sets the error flag.
#include "fl_mpnn.cuh"

namespace fl {

// ------------------------------------------------------------- column sums
// x[u] of lane l: row l, column u of a 32 x 32 block; returns the sum of
// column l over the rows, in a fixed tree order.
__device__ __forceinline__ float column_sums32(float (&x)[32], int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool hi = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < o; ++j) {
            const float send = hi ? x[j] : x[j + o];
            const float keep = hi ? x[j + o] : x[j];
            x[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return x[0];
}

__device__ __forceinline__ uint32_t positive_mask(uint32_t z) {  // 0xffff where a bf16 half is > 0
    const __nv_bfloat162 zero = __floats2bfloat162_rn(0.0f, 0.0f);
    return __hgt2_mask(*(const __nv_bfloat162 *)&z, zero);
}

// ------------------------------------------------------------- MLP backward
constexpr int MB_WARPS = 8, MB_THREADS = 32 * (MB_WARPS + 1);
constexpr int MB_CHUNKS = 8;
constexpr int MB_SMEM = MB_CHUNKS * MM_CHUNK_BYTES + 256 + 1024;

struct MlpBwdArgs {
    const float *dy;               // [M, ldy >= n2] fp32, or nullptr with dyb
    int64_t ldy;
    const __nv_bfloat16 *dyb;      // [M, 128] bf16 (n2 = 128): already rounded, its column sums already taken
    const __nv_bfloat16 *z;        // [M, 128] hidden activations
    const __nv_bfloat16 *w2t;      // [128, n2]
    const __nv_bfloat16 *w1t;      // [128 (decoder) or 256 (layer), 128]
    const __nv_bfloat16 *e2t;      // [128, 128] (layer)
    int64_t ldw2t, ldw1t, lde2t;
    __nv_bfloat16 *dz2;            // [M, n2] (with dy)
    __nv_bfloat16 *dz1;            // [M, 128]
    float *dx;                     // [M, 128] (decoder: dx; layer: dy + dx)
    __nv_bfloat16 *dagg;           // [M, 128] (layer)
    const int32_t *start;          // [M + 1] incoming edges (layer)
    const __nv_bfloat16 *z1e;      // [E, 128] (layer)
    __nv_bfloat16 *dze;            // [E, 128] (layer)
    float *cs_b2, *cs_b1, *cs_e2, *cs_e1;  // column sums, [4 x grid, n2 or 128] each
    int32_t n2, M;
    int32_t *error;
};

// MODE 0: encoder (no dx), 1: decoder, 2: processor layer.
// TMEM: 0 first product / message product, 128 dagg, 256 dx, 384 and 448 operands.
template <int MODE>
__global__ void __launch_bounds__(MB_THREADS, 1) k_mlp_bwd(const __grid_constant__ MlpBwdArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sW2 = smem_addr(smem), sW1 = sW2 + 2 * MM_CHUNK_BYTES, sE2 = sW1 + 4 * MM_CHUNK_BYTES;
    uint64_t *bars = (uint64_t *)(smem + MB_CHUNKS * MM_CHUNK_BYTES);
    const uint32_t in1 = smem_addr(bars), in2 = in1 + 8, in3 = in1 + 16, d1 = in1 + 24, d2a = in1 + 32, d2b = in1 + 40,
                   d3 = in1 + 48, drain = in1 + 56;
    uint32_t *tmem_slot = (uint32_t *)(bars + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = (g.M + MM_BM - 1) / MM_BM;
    const int k2 = g.n2 / 64;  // chunks of the first product
    if (tid == 0) {
        mbar_init(in1, MB_WARPS);
        mbar_init(in2, MB_WARPS);
        mbar_init(in3, MB_WARPS);
        mbar_init(d1, 1);
        mbar_init(d2a, 1);
        mbar_init(d2b, 1);
        mbar_init(d3, 1);
        mbar_init(drain, 1);
        mbar_fence_init();
    }
    if (warp == MB_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    for (int c = 0; c < k2; ++c) load_weight_chunk(g.w2t, g.ldw2t, MF_H, c, sW2 + c * MM_CHUNK_BYTES, tid, MB_THREADS);
    if (MODE > 0) {
        for (int c = 0; c < 2; ++c) {
            load_weight_chunk(g.w1t, g.ldw1t, MF_H, c, sW1 + c * MM_CHUNK_BYTES, tid, MB_THREADS);
            if (MODE == 2) {
                load_weight_chunk(g.w1t + MF_H * g.ldw1t, g.ldw1t, MF_H, c, sW1 + (2 + c) * MM_CHUNK_BYTES, tid, MB_THREADS);
                load_weight_chunk(g.e2t, g.lde2t, MF_H, c, sE2 + c * MM_CHUNK_BYTES, tid, MB_THREADS);
            }
        }
    }
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

    if (warp == MB_WARPS) {
        const bool issuer = elect_one();
        const uint32_t idesc = umma_idesc_bf16_128x128();
        auto product = [&](uint32_t d, uint32_t a, uint32_t sB, int steps, uint32_t done) {
            for (int s = 0; s < steps; ++s)
                umma_bf16_ts(tmem + d, tmem + a + 8u * s, umma_desc_sw128(sB + (s >> 2) * MM_CHUNK_BYTES + (s & 3) * 32),
                             idesc, s > 0);
            umma_commit(done);
        };
        int i = 0;
        for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x, ++i) {
            if (!warp_wait(in1, i & 1)) {
                bad = true;
                break;
            }
            tmem_fence_after();
            if (issuer) product(0, 384, sW2, 4 * k2, d1);
            if (MODE > 0) {
                if (!warp_wait(in2, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
                if (issuer) {
                    if (MODE == 2) product(128, 384, sW1 + 2 * MM_CHUNK_BYTES, 8, d2a);
                    product(256, 384, sW1, 8, d2b);
                }
            }
            if (MODE == 2) {
                if (!warp_wait(in3, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
                if (issuer) product(0, 448, sE2, 8, d3);
            }
        }
        if (issuer) umma_commit(drain);
        (void)warp_wait(drain, 0);
    } else {
        // thread = one row, 64 of its 128 columns
        const int quad = warp & 3, half = warp >> 2;
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        const int col = half * 64;
        float s_b2[2] = {0.0f, 0.0f}, s_b1[2] = {0.0f, 0.0f}, s_e2[2] = {0.0f, 0.0f}, s_e1[2] = {0.0f, 0.0f};
        auto hand_over = [&](uint32_t bar) {  // this warp's operand columns are written
            tmem_wait_st();
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        int i = 0;
        for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x, ++i) {
            const int r = t * MM_BM + quad * 32 + lane;
            const bool in = r < g.M;
            int rs = 0, deg = 0;
            if (MODE == 2 && in) {
                rs = g.start[r];
                deg = g.start[r + 1] - rs;
            }
            // dy -> bf16
            if (g.dy) {
                if (col < g.n2) {
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        float x[32];
                        uint32_t w[16];
#pragma unroll
                        for (int u = 0; u < 32; ++u) x[u] = 0.0f;
                        if (in) {
#pragma unroll
                            for (int u = 0; u < 32; u += 8) ld8f(g.dy + (int64_t)r * g.ldy + col + hh * 32 + u, x + u);
                        }
#pragma unroll
                        for (int u = 0; u < 16; ++u) w[u] = pack_bf16x2(x[2 * u], x[2 * u + 1]);
                        if (in) {
                            __nv_bfloat16 *p = g.dz2 + (int64_t)r * g.n2 + col + hh * 32;
                            st8u(p, w);
                            st8u(p + 16, w + 8);
                        }
                        __syncwarp();
                        tmem_st16(lanes + 384u + (uint32_t)(half * 32 + hh * 16), w);
                        s_b2[hh] += column_sums32(x, lane);
                    }
                }
            } else {
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t w[16];
#pragma unroll
                    for (int u = 0; u < 16; ++u) w[u] = 0u;
                    if (in) {
                        const __nv_bfloat16 *p = g.dyb + (int64_t)r * MF_H + col + hh * 32;
                        ld8u(p, w);
                        ld8u(p + 16, w + 8);
                    }
                    __syncwarp();
                    tmem_st16(lanes + 384u + (uint32_t)(half * 32 + hh * 16), w);
                }
            }
            hand_over(in1);
            // dz1 = relu'(z) (dz2 W2)
            {
                uint32_t zz[32];
#pragma unroll
                for (int u = 0; u < 32; ++u) zz[u] = 0u;
                if (in) {
#pragma unroll
                    for (int u = 0; u < 32; u += 8) ld8u(g.z + (int64_t)r * MF_H + col + 2 * u, zz + u);
                }
                if (!warp_wait(d1, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t v[32], w[16];
                    tmem_ld32(lanes + (uint32_t)(col + hh * 32), v);
                    float x[32];
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        const uint32_t m = positive_mask(zz[hh * 16 + u]);
                        x[2 * u] = (m & 0xffffu) ? __uint_as_float(v[2 * u]) : 0.0f;
                        x[2 * u + 1] = (m >> 16) ? __uint_as_float(v[2 * u + 1]) : 0.0f;
                        w[u] = pack_bf16x2(x[2 * u], x[2 * u + 1]);
                    }
                    if (in) {
                        __nv_bfloat16 *p = g.dz1 + (int64_t)r * MF_H + col + hh * 32;
                        st8u(p, w);
                        st8u(p + 16, w + 8);
                    }
                    __syncwarp();
                    if (MODE > 0) tmem_st16(lanes + 384u + (uint32_t)(half * 32 + hh * 16), w);
                    s_b1[hh] += column_sums32(x, lane);
                }
            }
            if (MODE == 0) {
                tmem_fence_before();
                continue;
            }
            hand_over(in2);
            if (MODE == 2) {
                // the message gradient, rounded; its sum over the cell's edges for the bias
                if (!warp_wait(d2a, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t v[32], w[16];
                    tmem_ld32(lanes + 128u + (uint32_t)(col + hh * 32), v);
                    float x[32];
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        const float a = __uint_as_float(v[2 * u]), b = __uint_as_float(v[2 * u + 1]);
                        w[u] = pack_bf16x2(a, b);
                        x[2 * u] = in ? a * (float)deg : 0.0f;
                        x[2 * u + 1] = in ? b * (float)deg : 0.0f;
                    }
                    if (in) {
                        __nv_bfloat16 *p = g.dagg + (int64_t)r * MF_H + col + hh * 32;
                        st8u(p, w);
                        st8u(p + 16, w + 8);
                    }
                    __syncwarp();
                    tmem_st16(lanes + 448u + (uint32_t)(half * 32 + hh * 16), w);
                    s_e2[hh] += column_sums32(x, lane);
                }
                hand_over(in3);
            }
            // dx (a layer: on top of dy, the residual's share)
            float o[32];
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                if (MODE == 2 && in) {
#pragma unroll
                    for (int u = 0; u < 32; u += 8) ld8f(g.dy + (int64_t)r * g.ldy + col + hh * 32 + u, o + u);
                }
                if (hh == 0) {
                    if (!warp_wait(d2b, i & 1)) {
                        bad = true;
                        break;
                    }
                    tmem_fence_after();
                }
                __syncwarp();
                uint32_t v[32];
                tmem_ld32(lanes + 256u + (uint32_t)(col + hh * 32), v);
                if (in) {
                    float x[32];
#pragma unroll
                    for (int u = 0; u < 32; ++u) x[u] = MODE == 2 ? o[u] + __uint_as_float(v[u]) : __uint_as_float(v[u]);
#pragma unroll
                    for (int u = 0; u < 32; u += 8) st8f(g.dx + (int64_t)r * MF_H + col + hh * 32 + u, x + u);
                }
                __syncwarp();
            }
            if (bad) break;
            if (MODE == 2) {
                // dz_e of the cell's edges
                if (!warp_wait(d3, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t v[32], w[16];
                    tmem_ld32(lanes + (uint32_t)(col + hh * 32), v);
                    float x[32];
#pragma unroll
                    for (int u = 0; u < 32; ++u) x[u] = 0.0f;
#pragma unroll
                    for (int u = 0; u < 16; ++u) w[u] = pack_bf16x2(__uint_as_float(v[2 * u]), __uint_as_float(v[2 * u + 1]));
#pragma unroll 1
                    for (int k = 0; k < 3; ++k) {
                        if (k < deg) {
                            const int64_t at = (int64_t)(rs + k) * MF_H + col + hh * 32;
                            uint32_t m[16];
                            ld8u(g.z1e + at, m);
                            ld8u(g.z1e + at + 16, m + 8);
#pragma unroll
                            for (int u = 0; u < 16; ++u) {
                                m[u] = positive_mask(m[u]);
                                if (m[u] & 0xffffu) x[2 * u] += __uint_as_float(v[2 * u]);
                                if (m[u] >> 16) x[2 * u + 1] += __uint_as_float(v[2 * u + 1]);
                                m[u] &= w[u];
                            }
                            st8u(g.dze + at, m);
                            st8u(g.dze + at + 16, m + 8);
                        }
                    }
                    __syncwarp();
                    s_e1[hh] += column_sums32(x, lane);
                }
            }
            tmem_fence_before();
        }
        const int64_t row = (int64_t)blockIdx.x * 4 + quad;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int c = col + hh * 32 + lane;
            if (g.dy && col < g.n2) g.cs_b2[row * g.n2 + c] = s_b2[hh];
            g.cs_b1[row * MF_H + c] = s_b1[hh];
            if (MODE == 2) {
                g.cs_e2[row * MF_H + c] = s_e2[hh];
                g.cs_e1[row * MF_H + c] = s_e1[hh];
            }
        }
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    tmem_fence_before();
    __syncthreads();
    if (warp == MB_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ------------------------------------------------------------- edge input gradients
constexpr int EB_PROD = 2, EB_EPI = 8, EB_THREADS = 32 * (EB_PROD + 1 + EB_EPI);
constexpr int EB_RING = 9;
constexpr int EB_SMEM = (4 + EB_RING) * MM_CHUNK_BYTES + 512 + 1024;

struct EdgeBwdArgs {
    const __nv_bfloat16 *dze;       // [E, 128]
    const __nv_bfloat16 *w1t;       // [256 of 384, 128]: rows of the receiver's, then of the sender's columns
    int64_t ldw1t;
    const int32_t *start;           // [C + 1] incoming edges e = start[c] ..
    const int32_t *send_start, *send_order;  // outgoing edges send_order[send_start[c] ..]
    float *dh;                      // [C, 128], updated
    int32_t C;
    int32_t *error;
};

// A producer warp's 64 rows of a 128-row chunk; own0 / own1: this lane's rows
// (lane, lane + 32), nullptr: left as it is.
__device__ __forceinline__ void warp_copy_rows64(const __nv_bfloat16 *own0, const __nv_bfloat16 *own1, uint32_t sdst, int pw,
                                                 int lane) {
    const int c = lane & 7;
    const uint64_t p0 = (uint64_t)own0, p1 = (uint64_t)own1;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int rr = 4 * i + (lane >> 3);
        const uint64_t row = __shfl_sync(0xffffffffu, i < 8 ? p0 : p1, rr & 31);
        const int R = 64 * pw + rr;
        if (row) cp_async16(sdst + (uint32_t)(R * 128 + ((c ^ (R & 7)) << 4)), (const __nv_bfloat16 *)row + c * 8);
    }
}

// Products p = 0..2: incoming slots, 3..5: outgoing slots of 128 cells; four
// 128-column TMEM regions in turn.
__global__ void __launch_bounds__(EB_THREADS, 1) k_edge_bwd(const __grid_constant__ EdgeBwdArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sW = smem_addr(smem), sR = sW + 4 * MM_CHUNK_BYTES;
    uint64_t *bars = (uint64_t *)(smem + (4 + EB_RING) * MM_CHUNK_BYTES);
    const uint32_t ringf = smem_addr(bars), ringe = ringf + 8 * EB_RING, df = ringe + 8 * EB_RING, de = df + 32, drain = de + 32;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * EB_RING + 4 + 4 + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = (g.C + MM_BM - 1) / MM_BM;
    if (tid == 0) {
        for (int s = 0; s < EB_RING; ++s) {
            mbar_init(ringf + 8 * s, 32 * EB_PROD);
            mbar_init(ringe + 8 * s, 1);
        }
        for (int k = 0; k < 4; ++k) {
            mbar_init(df + 8 * k, 1);
            mbar_init(de + 8 * k, EB_EPI);
        }
        mbar_init(drain, 1);
        mbar_fence_init();
    }
    if (warp == EB_PROD) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    for (int c = 0; c < 4; ++c)  // chunk = 64 K columns of 128 rows: receiver part 0, 1, sender part 0, 1
        load_weight_chunk(g.w1t + (c >> 1) * MF_H * g.ldw1t, g.ldw1t, MF_H, c & 1, sW + c * MM_CHUNK_BYTES, tid, EB_THREADS);
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

    if (warp < EB_PROD) {
        int q = 0;
        int t = blockIdx.x;
        // per lane two rows: first edge, edge counts (incoming, outgoing), outgoing edges
        int rs[2], deg[2], so[2], sdeg[2], ord[2][3];
        auto load_starts = [&](int tt, int (&a)[2], int (&b)[2], int (&c)[2], int (&d)[2]) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int cell = tt * MM_BM + 64 * warp + lane + 32 * j;
                a[j] = b[j] = c[j] = d[j] = 0;
                if (tt < tiles && cell < g.C) {
                    a[j] = g.start[cell];
                    b[j] = g.start[cell + 1] - a[j];
                    c[j] = g.send_start[cell];
                    d[j] = g.send_start[cell + 1] - c[j];
                }
            }
        };
        auto load_orders = [&](const int (&c)[2], const int (&d)[2], int (&o)[2][3]) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int k = 0; k < 3; ++k) o[j][k] = k < d[j] ? g.send_order[c[j] + k] : -1;
        };
        load_starts(t, rs, deg, so, sdeg);
        load_orders(so, sdeg, ord);
        for (; t < tiles && !bad;) {
            const int tn = t + gridDim.x;
            int nrs[2], ndeg[2], nso[2], nsd[2], nord[2][3];
            load_starts(tn, nrs, ndeg, nso, nsd);  // the next tile's, used in the next round
#pragma unroll
            for (int p = 0; p < 6; ++p) {
                const __nv_bfloat16 *row[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int e = p < 3 ? (p < deg[j] ? rs[j] + p : -1) : ord[j][p - 3 < 0 ? 0 : p - 3];
                    row[j] = e >= 0 ? g.dze + (int64_t)e * MF_H : nullptr;
                }
                if (p == 3) load_orders(nso, nsd, nord);
#pragma unroll 1
                for (int c = 0; c < 2; ++c, ++q) {
                    const int s = q % EB_RING, u = q / EB_RING;
                    if (u > 0 && !warp_wait(ringe + 8 * s, (u - 1) & 1)) {
                        bad = true;
                        break;
                    }
                    warp_copy_rows64(row[0] ? row[0] + c * 64 : nullptr, row[1] ? row[1] + c * 64 : nullptr,
                                     sR + s * MM_CHUNK_BYTES, warp, lane);
                    cp_async_arrive_noinc(ringf + 8 * s);
                }
                if (bad) break;
            }
            t = tn;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                rs[j] = nrs[j];
                deg[j] = ndeg[j];
#pragma unroll
                for (int k = 0; k < 3; ++k) ord[j][k] = nord[j][k];
            }
        }
        cp_async_wait_all();
    } else if (warp == EB_PROD) {
        const bool issuer = elect_one();
        const uint32_t idesc = umma_idesc_bf16_128x128();
        int q = 0, m = 0;
        for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x) {
            for (int p = 0; p < 6 && !bad; ++p, ++m) {
                const int reg = m & 3;
                if (m >= 4 && !warp_wait(de + 8 * reg, ((m >> 2) - 1) & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
                for (int c = 0; c < 2; ++c, ++q) {
                    const int st = q % EB_RING;
                    if (!warp_wait(ringf + 8 * st, (q / EB_RING) & 1)) {
                        bad = true;
                        break;
                    }
                    fence_async_smem();
                    if (issuer) {
                        const uint32_t a0 = sR + st * MM_CHUNK_BYTES, b0 = sW + ((p < 3 ? 0 : 2) + c) * MM_CHUNK_BYTES;
#pragma unroll
                        for (int s = 0; s < 4; ++s)
                            umma_bf16(tmem + 128u * reg, umma_desc_sw128(a0 + s * 32), umma_desc_sw128(b0 + s * 32), idesc,
                                      (c > 0 || s > 0) ? 1u : 0u);
                        umma_commit(ringe + 8 * st);
                    }
                }
                if (bad) break;
                if (issuer) umma_commit(df + 8 * reg);
            }
        }
        if (issuer) umma_commit(drain);
        (void)warp_wait(drain, 0);
    } else {
        // thread = one cell, 64 of its 128 columns
        const int quad = warp & 3, half = (warp - EB_PROD - 1) >> 2;
        const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * 64);
        int m = 0;
        for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x) {
            const int c = t * MM_BM + quad * 32 + lane;
            const bool in = c < g.C;
            int deg = 0, sdeg = 0;
            float tot[64], acc[64];
            float *row = g.dh + (int64_t)c * MF_H + half * 64;
            if (in) {
                deg = g.start[c + 1] - g.start[c];
                sdeg = g.send_start[c + 1] - g.send_start[c];
#pragma unroll
                for (int u = 0; u < 64; u += 8) ld8f(row + u, tot + u);
            }
#pragma unroll
            for (int p = 0; p < 6; ++p, ++m) {
                if (!warp_wait(df + 8 * (m & 3), (m >> 2) & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
                const bool valid = p < 3 ? p < deg : p - 3 < sdeg;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    uint32_t v[16];
                    tmem_ld16(base + 128u * (m & 3) + 16u * b, v);
                    if (b == 3) {
                        tmem_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(de + 8 * (m & 3));
                    }
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        const float a = (p == 0 || p == 3) ? 0.0f : acc[b * 16 + u];
                        acc[b * 16 + u] = valid ? a + __uint_as_float(v[u]) : a;
                        if (p == 2 || p == 5) tot[b * 16 + u] = acc[b * 16 + u] + tot[b * 16 + u];
                    }
                }
            }
            if (bad) break;
            if (in) {
#pragma unroll
                for (int u = 0; u < 64; u += 8) st8f(row + u, tot + u);
            }
            __syncwarp();
        }
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    tmem_fence_before();
    __syncthreads();
    if (warp == EB_PROD) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ------------------------------------------------------------- edge encoder's output gradient
constexpr int ES_PROD = 2, ES_EPI = 16, ES_THREADS = 32 * (ES_PROD + 1 + ES_EPI);
constexpr int ES_RING = 4, ES_STAGE = 3 * MM_CHUNK_BYTES, ES_MAX_LAYERS = 32;
constexpr int ES_SMEM = ES_RING * ES_STAGE + 256 + 1024;

struct EdgeSumArgs {
    const __nv_bfloat16 *dze[ES_MAX_LAYERS];  // [E, 128], in the order of the sum
    const __nv_bfloat16 *wt[ES_MAX_LAYERS];   // [128, ldwt]: rows = the edge features' columns of the weight
    int64_t ldwt[ES_MAX_LAYERS];
    __nv_bfloat16 *out;                        // [E, 128] bf16
    float *cs;                                 // column sums of the fp32 values, [8 x grid, 128]
    int32_t layers, E;
    int32_t *error;
};

// 256 rows a step (two row tiles), so a weight chunk serves both.  Each
// layer's product is a TMEM accumulator of its own (two buffers); the layers
// are added in fp32 in registers, in their order.
__global__ void __launch_bounds__(ES_THREADS, 1) k_edge_dsum(const __grid_constant__ EdgeSumArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sR = smem_addr(smem);
    uint64_t *bars = (uint64_t *)(smem + ES_RING * ES_STAGE);
    const uint32_t ringf = smem_addr(bars), ringe = ringf + 8 * ES_RING, df = ringe + 8 * ES_RING, de = df + 16, drain = de + 16;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * ES_RING + 2 + 2 + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int steps = (g.E + 2 * MM_BM - 1) / (2 * MM_BM);
    if (tid == 0) {
        for (int s = 0; s < ES_RING; ++s) {
            mbar_init(ringf + 8 * s, 32 * ES_PROD);
            mbar_init(ringe + 8 * s, 1);
        }
        for (int k = 0; k < 2; ++k) {
            mbar_init(df + 8 * k, 1);
            mbar_init(de + 8 * k, ES_EPI);
        }
        mbar_init(drain, 1);
        mbar_fence_init();
    }
    if (warp == ES_PROD) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool bad = false;
    pdl_wait();
    pdl_launch_dependents();

    if (warp < ES_PROD) {
        int q = 0;
        const int R0 = 64 * warp + lane, R1 = R0 + 32;
        for (int t = blockIdx.x; t < steps && !bad; t += gridDim.x) {
            for (int c = 0; c < 2 * g.layers; ++c, ++q) {
                const int s = q % ES_RING, u = q / ES_RING;
                if (u > 0 && !warp_wait(ringe + 8 * s, (u - 1) & 1)) {
                    bad = true;
                    break;
                }
                const __nv_bfloat16 *z = g.dze[c >> 1] + (c & 1) * 64, *w = g.wt[c >> 1] + (c & 1) * 64;
                const uint32_t dst = sR + s * ES_STAGE;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int r0 = t * 2 * MM_BM + j * MM_BM + R0, r1 = r0 + 32;
                    warp_copy_rows64(r0 < g.E ? z + (int64_t)r0 * MF_H : nullptr, r1 < g.E ? z + (int64_t)r1 * MF_H : nullptr,
                                     dst + j * MM_CHUNK_BYTES, warp, lane);
                }
                warp_copy_rows64(w + (int64_t)R0 * g.ldwt[c >> 1], w + (int64_t)R1 * g.ldwt[c >> 1],
                                 dst + 2 * MM_CHUNK_BYTES, warp, lane);
                cp_async_arrive_noinc(ringf + 8 * s);
            }
        }
        cp_async_wait_all();
    } else if (warp == ES_PROD) {
        const bool issuer = elect_one();
        const uint32_t idesc = umma_idesc_bf16_128x128();
        int q = 0, n = 0;
        for (int t = blockIdx.x; t < steps && !bad; t += gridDim.x) {
            for (int l = 0; l < g.layers && !bad; ++l, ++n) {
                const int b = n & 1;
                if (n >= 2 && !warp_wait(de + 8 * b, ((n >> 1) - 1) & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
                for (int c = 0; c < 2; ++c, ++q) {
                    const int st = q % ES_RING;
                    if (!warp_wait(ringf + 8 * st, (q / ES_RING) & 1)) {
                        bad = true;
                        break;
                    }
                    fence_async_smem();
                    if (issuer) {
                        const uint32_t a0 = sR + st * ES_STAGE, b0 = a0 + 2 * MM_CHUNK_BYTES;
#pragma unroll
                        for (int j = 0; j < 2; ++j)
#pragma unroll
                            for (int s = 0; s < 4; ++s)
                                umma_bf16(tmem + (uint32_t)(b * 256 + j * 128), umma_desc_sw128(a0 + j * MM_CHUNK_BYTES + s * 32),
                                          umma_desc_sw128(b0 + s * 32), idesc, (c > 0 || s > 0) ? 1u : 0u);
                        umma_commit(ringe + 8 * st);
                    }
                }
                if (bad) break;
                if (issuer) umma_commit(df + 8 * b);
            }
        }
        if (issuer) umma_commit(drain);
        (void)warp_wait(drain, 0);
    } else {
        // thread = one row of one of the two tiles, 64 of its 128 columns
        const int quad = warp & 3, half = ((warp - ES_PROD - 1) >> 2) & 1, j = (warp - ES_PROD - 1) >> 3;
        const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(j * 128 + half * 64);
        float sum[2] = {0.0f, 0.0f};
        int n = 0;
        for (int t = blockIdx.x; t < steps && !bad; t += gridDim.x) {
            const int r = t * 2 * MM_BM + j * MM_BM + quad * 32 + lane;
            const bool in = r < g.E;
            float acc[2][32];
#pragma unroll
            for (int u = 0; u < 64; ++u) acc[u >> 5][u & 31] = 0.0f;
            for (int l = 0; l < g.layers; ++l, ++n) {
                const int b = n & 1;
                if (!warp_wait(df + 8 * b, (n >> 1) & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    uint32_t v[16];
                    tmem_ld16(base + (uint32_t)(b * 256 + k * 16), v);
                    if (k == 3) {
                        tmem_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(de + 8 * b);
                    }
                    if (in) {
#pragma unroll
                        for (int u = 0; u < 16; ++u) acc[k >> 1][(k & 1) * 16 + u] += __uint_as_float(v[u]);
                    }
                }
            }
            if (bad) break;
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                if (in) {
                    __nv_bfloat16 *p = g.out + (int64_t)r * MF_H + half * 64 + hh * 32;
#pragma unroll
                    for (int u = 0; u < 32; u += 16) {
                        uint32_t w[8];
#pragma unroll
                        for (int y = 0; y < 8; ++y) w[y] = pack_bf16x2(acc[hh][u + 2 * y], acc[hh][u + 2 * y + 1]);
                        st8u(p + u, w);
                    }
                }
                __syncwarp();
                sum[hh] += column_sums32(acc[hh], lane);
            }
        }
        const int64_t row = (int64_t)blockIdx.x * 8 + j * 4 + quad;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) g.cs[row * MF_H + half * 64 + hh * 32 + lane] = sum[hh];
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    tmem_fence_before();
    __syncthreads();
    if (warp == ES_PROD) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ------------------------------------------------------------- weight gradients
constexpr int WG_PROD = 8, WG_THREADS = 32 * (WG_PROD + 1), WG_JOBS = 4;
constexpr int WG_BLOCK = 64 * 128;                  // 64 rows x 64 columns of bf16
constexpr int WG_RING_BYTES = 224 * 1024, WG_MAX_RING = 7;
constexpr int WG_SMEM = WG_RING_BYTES + 256 + 1024;

struct WgSeg {
    const __nv_bfloat16 *base;
    const int32_t *rows;
    int64_t ld;
    int32_t width;                                  // 64 or 128
};

struct WgJob {
    WgSeg a, x[3];                                  // dZ (64 or 128 columns) and the segments of X
    int32_t nx, n_in, M;
    int32_t cta0, ctas;
    float *part;                                    // [ctas, a.width, n_in]
};

struct WgArgs {
    WgJob job[WG_JOBS];
    int32_t jobs;
    int32_t *error;
};

// Stage: 64 rows of dZ (two 64-column blocks of 8 KB) then of X's segments.
__global__ void __launch_bounds__(WG_THREADS, 1) k_wgrad(const __grid_constant__ WgArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sR = smem_addr(smem);
    uint64_t *bars = (uint64_t *)(smem + WG_RING_BYTES);
    const uint32_t ringf = smem_addr(bars), ringe = ringf + 8 * WG_MAX_RING, done = ringe + 8 * WG_MAX_RING;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * WG_MAX_RING + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int jn = 0;
    while (jn + 1 < g.jobs && (int)blockIdx.x >= g.job[jn + 1].cta0) ++jn;
    const WgJob &J = g.job[jn];
    const int li = (int)blockIdx.x - J.cta0;
    const int stage = (2 + J.n_in / 64) * WG_BLOCK, S = min(WG_MAX_RING, WG_RING_BYTES / stage);
    const int64_t chunks = (J.M + 63) / 64;
    const int c0 = (int)(chunks * li / J.ctas), c1 = (int)(chunks * (li + 1) / J.ctas);
    if (tid == 0) {
        for (int s = 0; s < WG_MAX_RING; ++s) {
            mbar_init(ringf + 8 * s, 32 * WG_PROD);
            mbar_init(ringe + 8 * s, 1);
        }
        mbar_init(done, 1);
        mbar_fence_init();
    }
    if (warp == WG_PROD) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (J.a.width == 64) {  // the upper 64 output rows do not exist: zero operand columns
        for (int s = 0; s < S; ++s)
            for (int p = tid; p < WG_BLOCK / 16; p += WG_THREADS)
                asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(sR + s * stage + WG_BLOCK + p * 16), "r"(0u) : "memory");
    }
    fence_async_smem();
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool bad = false;
    pdl_wait();
    pdl_launch_dependents();

    if (warp < WG_PROD) {
        // producers: 8 rows of each 64-row chunk (lanes 0..7 own one each);
        // row maps are read one chunk ahead.  The job's fields are held in
        // registers: read from the parameters in the copy loop they made it
        // 230 cycles an instruction
        const WgSeg G[4] = {J.a, J.x[0], J.x[1], J.x[2]};
        const int nx = J.nx, M = J.M, own = 8 * warp + (lane & 7), piece = lane & 7;
        uint32_t off[4];
        off[0] = 0;
        off[1] = 2 * WG_BLOCK;
        off[2] = off[1] + (G[1].width / 64) * WG_BLOCK;
        off[3] = off[2] + (G[2].width / 64) * WG_BLOCK;
        auto load_rows = [&](int c, const __nv_bfloat16 *(&o)[4]) {
            const int r = c * 64 + own;
            const bool in = c < c1 && r < M;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                o[x] = nullptr;
                if (in && x <= nx) o[x] = G[x].base + (G[x].rows ? (int64_t)G[x].rows[r] : (int64_t)r) * G[x].ld;
            }
        };
        const __nv_bfloat16 *row[4], *nrow[4];
        load_rows(c0, row);
        int s = 0, u = 0;
        for (int c = c0; c < c1 && !bad; ++c) {
            load_rows(c + 1, nrow);
            if (u > 0 && !warp_wait(ringe + 8 * s, (u - 1) & 1)) {
                bad = true;
                break;
            }
            const uint32_t dst = sR + s * stage;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                if (x <= nx) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int rr = 4 * i + (lane >> 3), R = 8 * warp + rr;
                        const __nv_bfloat16 *src = (const __nv_bfloat16 *)__shfl_sync(0xffffffffu, (uint64_t)row[x], rr);
                        const uint32_t d = dst + off[x] + (uint32_t)(R * 128 + ((piece ^ (R & 7)) << 4));
                        if (src) {
                            cp_async16(d, src + piece * 8);
                            if (G[x].width == 128) cp_async16(d + WG_BLOCK, src + 64 + piece * 8);
                        } else {
                            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(d), "r"(0u) : "memory");
                            if (G[x].width == 128)
                                asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(d + WG_BLOCK), "r"(0u) : "memory");
                        }
                    }
                }
            }
            cp_async_arrive_noinc(ringf + 8 * s);
#pragma unroll
            for (int x = 0; x < 4; ++x) row[x] = nrow[x];
            if (++s == S) {
                s = 0;
                ++u;
            }
        }
        cp_async_wait_all();
        // the partial product: thread = one output row
        if (!bad && !warp_wait(done, 0)) bad = true;
        if (!bad) {
            tmem_fence_after();
            const int r = (warp & 3) * 32 + lane;
            float *out = J.part + ((int64_t)li * J.a.width + r) * J.n_in;
            for (int cb = (warp >> 2) * 32; cb < J.n_in; cb += 64) {
                uint32_t v[32];
                tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)cb, v);
                if (r < J.a.width) {
#pragma unroll
                    for (int u = 0; u < 32; u += 8) st8u(out + cb + u, v + u);
                }
                __syncwarp();
            }
        }
    } else {
        const bool issuer = elect_one();
        // at most 256 columns an instruction: columns [0, w0) and [256, n_in)
        const int n_in = J.n_in, w0 = min(256, n_in);
        const uint32_t i0 = umma_idesc_bf16_mn(w0), i1 = umma_idesc_bf16_mn(n_in > 256 ? n_in - 256 : 64);
        int s = 0, ph = 0;
        uint32_t acc = 0u;
        for (int c = c0; c < c1 && !bad; ++c) {
            if (!warp_wait(ringf + 8 * s, ph)) {
                bad = true;
                break;
            }
            fence_async_smem();
            if (issuer) {
                const uint32_t a0 = sR + s * stage, x0 = a0 + 2 * WG_BLOCK;
#pragma unroll
                for (int k = 0; k < 4; ++k) {  // 16 rows each
                    const uint64_t da = umma_desc_mn_sw128(a0 + k * 2048, WG_BLOCK);
                    umma_bf16(tmem, da, umma_desc_mn_sw128(x0 + k * 2048, WG_BLOCK), i0, acc);
                    if (n_in > 256) umma_bf16(tmem + 256u, da, umma_desc_mn_sw128(x0 + 4 * WG_BLOCK + k * 2048, WG_BLOCK), i1, acc);
                    acc = 1u;
                }
                umma_commit(ringe + 8 * s);
            }
            if (++s == S) {
                s = 0;
                ph ^= 1;
            }
        }
        if (issuer) umma_commit(done);
        (void)warp_wait(done, 0);
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    tmem_fence_before();
    __syncthreads();
    if (warp == WG_PROD) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ------------------------------------------------------------- partial sums
constexpr int RD_JOBS = 12;

struct RdJob {
    const float *part;  // [count, n]
    float *out;         // [n], added to
    int32_t count, n;   // n a multiple of 4
};

struct RdArgs {
    RdJob job[RD_JOBS];
};

// Block (32, 8): 32 groups of four columns, each over eight interleaved
// subsets of the partials, combined in subset order.
__global__ void __launch_bounds__(256) k_reduce(const __grid_constant__ RdArgs g) {
    pdl_wait();
    pdl_launch_dependents();
    const RdJob &J = g.job[blockIdx.y];
    const int i = ((int)blockIdx.x * 32 + (int)threadIdx.x) * 4;
    __shared__ float4 red[8][32];
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (i < J.n) {
#pragma unroll 4
        for (int p = threadIdx.y; p < J.count; p += 8) {
            const float4 v = *(const float4 *)(J.part + (int64_t)p * J.n + i);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
    }
    red[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y || i >= J.n) return;
#pragma unroll
    for (int p = 1; p < 8; ++p) {
        const float4 v = red[p][threadIdx.x];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    float4 *o = (float4 *)(J.out + i);
    const float4 v = *o;
    *o = make_float4(v.x + s.x, v.y + s.y, v.z + s.z, v.w + s.w);
}

// ------------------------------------------------------------- optimizer
constexpr int AD_JOBS = 128;

struct AdJob {
    float *w, *m1, *m2;
    const float *g;
    __nv_bfloat16 *wb, *wt;
    int32_t rows, cols, ldt, block0;
};

struct AdArgs {
    AdJob job[AD_JOBS];
    float lr, b1, b2, eps, c1, c2, wd;
    int32_t jobs;
};

// One Adam step over all of a network's tensors (k_adam's arithmetic).
__global__ void __launch_bounds__(256) k_adam_all(const __grid_constant__ AdArgs g) {
    int lo = 0, hi = g.jobs;  // job[lo].block0 <= blockIdx.x < job[hi].block0
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (g.job[mid].block0 <= (int)blockIdx.x) lo = mid; else hi = mid;
    }
    const AdJob &J = g.job[lo];
    const int i = ((int)blockIdx.x - J.block0) * 256 + (int)threadIdx.x;
    if (i >= J.rows * J.cols) return;
    const float w0 = J.w[i], gi = J.g[i] + g.wd * w0;
    const float a = g.b1 * J.m1[i] + (1.0f - g.b1) * gi;
    const float b = g.b2 * J.m2[i] + (1.0f - g.b2) * gi * gi;
    J.m1[i] = a;
    J.m2[i] = b;
    const float wi = w0 - g.lr * (a / g.c1) / (sqrtf(b / g.c2) + g.eps);
    J.w[i] = wi;
    const __nv_bfloat16 h = __float2bfloat16(wi);
    if (J.wb) J.wb[i] = h;
    if (J.wt) {
        const int r = i / J.cols, c = i - r * J.cols;
        J.wt[(int64_t)c * J.ldt + r] = h;
    }
}

// floats of scratch that fl_mpnn_backward needs on a device of `sms` SMs: the
// weight gradients' partials (at most 128 x 384 per CTA) and eight sets of
// column sums (four rows of 128 per CTA).
static int64_t backward_scratch(int sms) { return (int64_t)sms * (MF_H * 3 * MF_H + 8 * 4 * MF_H); }

static cudaError_t current_sms(int *dev, int *sms) {
    cudaError_t e = cudaGetDevice(dev);
    return e == cudaSuccess ? cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, *dev) : e;
}

}  // namespace fl

using namespace fl;

extern "C" {

FL_API int fl_mpnn_backward_scratch(int64_t *floats) {
    if (!floats) return set_error(FL_E_INVALID, "fl_mpnn_backward_scratch: NULL output");
    int dev = 0, sms = 0;
    const cudaError_t e = current_sms(&dev, &sms);
    if (e != cudaSuccess) return set_error(FL_E_NO_DEVICE, "no usable CUDA device: %s", cudaGetErrorString(e));
    *floats = backward_scratch(sms);
    return FL_OK;
}

FL_API int fl_mpnn_backward(const FlMpnnBackwardDesc *d, void *stream) {
    if (!d || d->cells < 1 || d->edges < 0 || d->layers < 0 || d->layers > ES_MAX_LAYERS)
        return set_error(FL_E_INVALID, "fl_mpnn_backward: bad sizes (at most %d layers)", ES_MAX_LAYERS);
    const int C = d->cells, E = d->edges, L = d->layers;
    if (!d->x || !d->dy || !d->recv_start || !d->zn || !d->zd || !d->h_bf || !d->dh[0] || !d->dh[1] || !d->dz2c || !d->dz1c ||
        !d->dyb || !d->scratch ||
        (L > 0 && (!d->edge || !d->node || !d->agg || !d->z1n || !d->z1e || !d->dze || !d->dagg || !d->send_start)) ||
        (E > 0 && (!d->src || !d->dst || !d->send_order || !d->ef || !d->ze || !d->e || !d->dz2e)))
        return set_error(FL_E_INVALID, "fl_mpnn_backward: NULL pointer");
    if (d->ldx < 64 || d->ldx % 8 || d->lde < 64 || d->lde % 8 || d->ldy < 64 || d->ldy % 8)
        return set_error(FL_E_INVALID, "fl_mpnn_backward: leading dimensions must be multiples of 8 and at least 64");
    uintptr_t a16 = (uintptr_t)d->x | (uintptr_t)d->ef;
    uintptr_t a32 = (uintptr_t)d->dy | (uintptr_t)d->zn | (uintptr_t)d->ze | (uintptr_t)d->e | (uintptr_t)d->zd |
                    (uintptr_t)d->dh[0] | (uintptr_t)d->dh[1] | (uintptr_t)d->dz2c | (uintptr_t)d->dz1c | (uintptr_t)d->dagg |
                    (uintptr_t)d->dyb | (uintptr_t)d->dz2e | (uintptr_t)d->scratch;
    bool ok = true;
    auto dense = [&](const FlDenseGrad &r, int n_out) {
        a16 |= (uintptr_t)r.wt | (uintptr_t)r.gw | (uintptr_t)r.gb;
        ok = ok && r.wt && r.gw && r.gb && r.ldwt >= n_out && r.ldwt % 8 == 0;
    };
    for (const FlDenseGrad *r : {&d->enc_n[0], &d->enc_n[1], &d->enc_e[0], &d->enc_e[1], &d->dec[0]}) dense(*r, 128);
    dense(d->dec[1], 64);
    for (int l = 0; l < L && ok; ++l) {
        for (int j = 0; j < 2; ++j) {
            dense(d->edge[2 * l + j], 128);
            dense(d->node[2 * l + j], 128);
        }
        ok = ok && d->h_bf[l] && d->agg[l] && d->z1n[l] && (E == 0 || (d->z1e[l] && d->dze[l]));
        a32 |= (uintptr_t)d->h_bf[l] | (uintptr_t)d->agg[l] | (uintptr_t)d->z1n[l] | (uintptr_t)d->z1e[l] | (uintptr_t)d->dze[l];
    }
    if (!ok || !d->h_bf[L]) return set_error(FL_E_INVALID, "fl_mpnn_backward: bad layer");
    a32 |= (uintptr_t)d->h_bf[L];
    if (a16 % 16 || a32 % 32)
        return set_error(FL_E_INVALID, "fl_mpnn_backward: inputs, weights and gradients must be 16-byte, buffers 32-byte aligned");
    int32_t *err = nullptr;
    int rc = gemm_error_flag(&err);
    if (rc) return rc;
    int dev = 0, sms = 0;
    cudaError_t e = current_sms(&dev, &sms);
    if (e == cudaSuccess && d->scratch_floats < backward_scratch(sms))
        return set_error(FL_E_INVALID, "fl_mpnn_backward: scratch of %lld floats, %lld needed", (long long)d->scratch_floats,
                         (long long)backward_scratch(sms));
    static std::atomic<uint64_t> done[6];
    if (e == cudaSuccess) e = allow_smem((const void *)k_mlp_bwd<0>, MB_SMEM, dev, done[0]);
    if (e == cudaSuccess) e = allow_smem((const void *)k_mlp_bwd<1>, MB_SMEM, dev, done[1]);
    if (e == cudaSuccess) e = allow_smem((const void *)k_mlp_bwd<2>, MB_SMEM, dev, done[2]);
    if (e == cudaSuccess) e = allow_smem((const void *)k_edge_bwd, EB_SMEM, dev, done[3]);
    if (e == cudaSuccess) e = allow_smem((const void *)k_edge_dsum, ES_SMEM, dev, done[4]);
    if (e == cudaSuccess) e = allow_smem((const void *)k_wgrad, WG_SMEM, dev, done[5]);
    cudaStream_t st = (cudaStream_t)stream;
    using bf = __nv_bfloat16;
    int64_t launched = 0;
    float *part = d->scratch, *cs[8];
    for (int k = 0; k < 8; ++k) cs[k] = part + (int64_t)sms * (MF_H * 3 * MF_H + k * 4 * MF_H);
    const int c_tiles = (C + MM_BM - 1) / MM_BM, e_tiles = (E + MM_BM - 1) / MM_BM;
    const int c_grid = std::min(c_tiles, sms), e_grid = std::max(1, std::min(e_tiles, sms));

    // the weight gradients of up to four products in one launch, the CTAs
    // shared out by the bytes each product stages; then every partial sum
    RdArgs rd;
    int n_rd = 0, rd_cols = 0;
    auto sums = [&](const float *p, int count, int n, float *out) {
        rd.job[n_rd++] = RdJob{p, out, count, n};
        rd_cols = std::max(rd_cols, n);
    };
    WgArgs wg;
    wg.jobs = 0;
    wg.error = err;
    float *wg_out[WG_JOBS];
    auto seg = [](const void *p, const int32_t *rows, int64_t ld, int width) { return WgSeg{(const bf *)p, rows, ld, width}; };
    auto product = [&](int M, WgSeg a, std::initializer_list<WgSeg> xs, float *gw) {
        if (M < 1) return;
        WgJob &J = wg.job[wg.jobs];
        J = WgJob{};
        J.a = a;
        J.M = M;
        for (const WgSeg &x : xs) {
            J.x[J.nx++] = x;
            J.n_in += x.width;
        }
        wg_out[wg.jobs++] = gw;
    };
    auto flush = [&]() {
        if (e != cudaSuccess) return;
        double total = 0.0;
        for (int j = 0; j < wg.jobs; ++j) total += (double)wg.job[j].M * (wg.job[j].a.width + wg.job[j].n_in);
        int cta = 0;
        float *p = part;
        for (int j = 0; j < wg.jobs; ++j) {
            WgJob &J = wg.job[j];
            const int left = wg.jobs - 1 - j, chunks = (J.M + 63) / 64;
            const double cost = (double)J.M * (J.a.width + J.n_in);
            int n = (int)(sms * cost / total + 0.5);
            n = std::max(1, std::min(std::min(n, chunks), sms - cta - left));
            J.cta0 = cta;
            J.ctas = n;
            J.part = p;
            cta += n;
            p += (int64_t)n * J.a.width * J.n_in;
            sums(J.part, n, J.a.width * J.n_in, wg_out[j]);
        }
        e = launch_blocks(k_wgrad, wg, cta, sms, WG_THREADS, WG_SMEM, launched > 0, st);
        ++launched;
        if (e == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)((rd_cols + 127) / 128), (unsigned)n_rd);
            cfg.blockDim = dim3(32, 8);
            cfg.stream = st;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            e = cudaLaunchKernelEx(&cfg, k_reduce, rd);
            ++launched;
        }
        wg.jobs = n_rd = rd_cols = 0;
    };
    auto mlp = [&](auto kernel, MlpBwdArgs a, int blocks) {
        if (e != cudaSuccess) return;
        a.error = err;
        e = launch_blocks(kernel, a, blocks, sms, MB_THREADS, MB_SMEM, launched > 0, st);
        ++launched;
    };

    // decoder
    {
        MlpBwdArgs a{};
        a.dy = d->dy;
        a.ldy = d->ldy;
        a.z = (const bf *)d->zd;
        a.w2t = (const bf *)d->dec[1].wt;
        a.ldw2t = d->dec[1].ldwt;
        a.w1t = (const bf *)d->dec[0].wt;
        a.ldw1t = d->dec[0].ldwt;
        a.dz2 = (bf *)d->dyb;
        a.dz1 = (bf *)d->dz1c;
        a.dx = d->dh[0];
        a.cs_b2 = cs[0];
        a.cs_b1 = cs[1];
        a.n2 = 64;
        a.M = C;
        mlp(k_mlp_bwd<1>, a, c_tiles);
        sums(cs[0], 4 * c_grid, 64, d->dec[1].gb);
        sums(cs[1], 4 * c_grid, MF_H, d->dec[0].gb);
        product(C, seg(d->dyb, nullptr, 64, 64), {seg(d->zd, nullptr, MF_H, MF_H)}, d->dec[1].gw);
        product(C, seg(d->dz1c, nullptr, MF_H, MF_H), {seg(d->h_bf[L], nullptr, MF_H, MF_H)}, d->dec[0].gw);
        flush();
    }
    int cur = 0;
    for (int l = L - 1; l >= 0 && e == cudaSuccess; --l, cur ^= 1) {
        const FlDenseGrad &e1 = d->edge[2 * l], &e2 = d->edge[2 * l + 1], &n1 = d->node[2 * l], &n2 = d->node[2 * l + 1];
        MlpBwdArgs a{};
        a.dy = d->dh[cur];
        a.ldy = MF_H;
        a.z = (const bf *)d->z1n[l];
        a.w2t = (const bf *)n2.wt;
        a.ldw2t = n2.ldwt;
        a.w1t = (const bf *)n1.wt;
        a.ldw1t = n1.ldwt;
        a.e2t = (const bf *)e2.wt;
        a.lde2t = e2.ldwt;
        a.dz2 = (bf *)d->dz2c;
        a.dz1 = (bf *)d->dz1c;
        a.dx = d->dh[cur ^ 1];
        a.dagg = (bf *)d->dagg;
        a.start = d->recv_start;
        a.z1e = (const bf *)d->z1e[l];
        a.dze = (bf *)d->dze[l];
        a.cs_b2 = cs[0];
        a.cs_b1 = cs[1];
        a.cs_e2 = cs[2];
        a.cs_e1 = cs[3];
        a.n2 = MF_H;
        a.M = C;
        mlp(k_mlp_bwd<2>, a, c_tiles);
        if (e == cudaSuccess && E > 0) {
            EdgeBwdArgs b{};
            b.dze = (const bf *)d->dze[l];
            b.w1t = (const bf *)e1.wt;
            b.ldw1t = e1.ldwt;
            b.start = d->recv_start;
            b.send_start = d->send_start;
            b.send_order = d->send_order;
            b.dh = d->dh[cur ^ 1];
            b.C = C;
            b.error = err;
            e = launch_blocks(k_edge_bwd, b, c_tiles, sms, EB_THREADS, EB_SMEM, true, st);
            ++launched;
        }
        sums(cs[0], 4 * c_grid, MF_H, n2.gb);
        sums(cs[1], 4 * c_grid, MF_H, n1.gb);
        sums(cs[2], 4 * c_grid, MF_H, e2.gb);
        sums(cs[3], 4 * c_grid, MF_H, e1.gb);
        product(E, seg(d->dze[l], nullptr, MF_H, MF_H),
                {seg(d->h_bf[l], d->dst, MF_H, MF_H), seg(d->h_bf[l], d->src, MF_H, MF_H), seg(d->e, nullptr, MF_H, MF_H)}, e1.gw);
        product(E, seg(d->dagg, d->dst, MF_H, MF_H), {seg(d->z1e[l], nullptr, MF_H, MF_H)}, e2.gw);
        product(C, seg(d->dz1c, nullptr, MF_H, MF_H),
                {seg(d->h_bf[l], nullptr, MF_H, MF_H), seg(d->agg[l], nullptr, MF_H, MF_H)}, n1.gw);
        product(C, seg(d->dz2c, nullptr, MF_H, MF_H), {seg(d->z1n[l], nullptr, MF_H, MF_H)}, n2.gw);
        flush();
    }
    // encoders
    {
        MlpBwdArgs a{};
        a.dy = d->dh[cur];
        a.ldy = MF_H;
        a.z = (const bf *)d->zn;
        a.w2t = (const bf *)d->enc_n[1].wt;
        a.ldw2t = d->enc_n[1].ldwt;
        a.dz2 = (bf *)d->dz2c;
        a.dz1 = (bf *)d->dz1c;
        a.cs_b2 = cs[0];
        a.cs_b1 = cs[1];
        a.n2 = MF_H;
        a.M = C;
        mlp(k_mlp_bwd<0>, a, c_tiles);
        sums(cs[0], 4 * c_grid, MF_H, d->enc_n[1].gb);
        sums(cs[1], 4 * c_grid, MF_H, d->enc_n[0].gb);
        product(C, seg(d->dz2c, nullptr, MF_H, MF_H), {seg(d->zn, nullptr, MF_H, MF_H)}, d->enc_n[1].gw);
        product(C, seg(d->dz1c, nullptr, MF_H, MF_H), {seg(d->x, nullptr, d->ldx, 64)}, d->enc_n[0].gw);
    }
    if (L > 0 && E > 0) {  // (without layers nothing depends on the edges)
        if (e == cudaSuccess) {
            EdgeSumArgs b{};
            for (int k = 0; k < L; ++k) {  // last layer first
                const int l = L - 1 - k;
                b.dze[k] = (const bf *)d->dze[l];
                b.wt[k] = (const bf *)d->edge[2 * l].wt + 2 * MF_H * d->edge[2 * l].ldwt;
                b.ldwt[k] = d->edge[2 * l].ldwt;
            }
            b.out = (bf *)d->dz2e;
            b.cs = cs[4];
            b.layers = L;
            b.E = E;
            b.error = err;
            e = launch_blocks(k_edge_dsum, b, (E + 2 * MM_BM - 1) / (2 * MM_BM), sms, ES_THREADS, ES_SMEM, true, st);
            ++launched;
        }
        MlpBwdArgs a{};
        a.dyb = (const bf *)d->dz2e;
        a.z = (const bf *)d->ze;
        a.w2t = (const bf *)d->enc_e[1].wt;
        a.ldw2t = d->enc_e[1].ldwt;
        a.dz1 = (bf *)d->dze[0];  // (no longer needed)
        a.cs_b1 = cs[6];
        a.n2 = MF_H;
        a.M = E;
        mlp(k_mlp_bwd<0>, a, e_tiles);
        sums(cs[4], 8 * std::min((E + 2 * MM_BM - 1) / (2 * MM_BM), sms), MF_H, d->enc_e[1].gb);  // (sets 4 and 5)
        sums(cs[6], 4 * e_grid, MF_H, d->enc_e[0].gb);
        product(E, seg(d->dz2e, nullptr, MF_H, MF_H), {seg(d->ze, nullptr, MF_H, MF_H)}, d->enc_e[1].gw);
        product(E, seg(d->dze[0], nullptr, MF_H, MF_H), {seg(d->ef, nullptr, d->lde, 64)}, d->enc_e[0].gw);
    }
    flush();
    if (e != cudaSuccess) return set_error(FL_E_CUDA, "fl_mpnn_backward: %s", cudaGetErrorString(e));
    add_launches(launched);
    return FL_OK;
}

FL_API int fl_adam_all(const FlAdamTensor *t, int32_t n, float lr, float b1, float b2, float eps, int32_t step,
                       float weight_decay, void *stream) {
    if (!t || n < 1 || step < 1) return set_error(FL_E_INVALID, "fl_adam_all: bad arguments");
    for (int k = 0; k < n; ++k)
        if (!t[k].w || !t[k].m1 || !t[k].m2 || !t[k].g || t[k].rows < 1 || t[k].cols < 1 ||
            (int64_t)t[k].rows * t[k].cols > (1 << 30) || (t[k].wt_bf16 && t[k].ldt < t[k].rows))
            return set_error(FL_E_INVALID, "fl_adam_all: tensor %d: bad arguments", k);
    AdArgs a;
    a.lr = lr;
    a.b1 = b1;
    a.b2 = b2;
    a.eps = eps;
    a.c1 = 1.0f - powf(b1, (float)step);
    a.c2 = 1.0f - powf(b2, (float)step);
    a.wd = weight_decay;
    for (int k0 = 0; k0 < n; k0 += AD_JOBS) {
        int blocks = 0;
        a.jobs = std::min(AD_JOBS, n - k0);
        for (int k = 0; k < a.jobs; ++k) {
            const FlAdamTensor &s = t[k0 + k];
            a.job[k] = AdJob{s.w, s.m1, s.m2, s.g, (__nv_bfloat16 *)s.w_bf16, (__nv_bfloat16 *)s.wt_bf16,
                             s.rows, s.cols, s.ldt, blocks};
            blocks += (int)(((int64_t)s.rows * s.cols + 255) / 256);
        }
        k_adam_all<<<blocks, 256, 0, (cudaStream_t)stream>>>(a);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return set_error(FL_E_CUDA, "k_adam_all launch: %s", cudaGetErrorString(e));
        add_launches(1);
    }
    return FL_OK;
}

}  // extern "C"
