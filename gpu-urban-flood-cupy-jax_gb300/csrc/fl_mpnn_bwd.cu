// The surrogate network's backward pass as fused blocks on the tensor cores:
//   k_mlp_bwd    a two-layer MLP's backward over rows: dz2 = bf16(dy), dz1 =
//                relu'(z) (dz2 W2), dx = dz1 W1; for a processor layer also dh = dy + dx, the message gradient
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
//                no transposed copies.  Rows are split into short partial
//                sums, the splits shared out over the CTAs
//   k_reduce     the partial sums, in order, into the gradients, and the fp32
//                column sums of the bias gradients by row class (mod 256)
//   k_bias_final the class sums, in order, into the bias gradients
// Everything keeps the rounding points and the orders of sums of the separate
// products (same bits): a bias that differs in its last bit moves some
// activation across a bf16 boundary every few steps, and a training run then
// goes its own way.  The message layers' second bias is the caller's.
//
// Measured: one optimizer step on 99,904 cells and 299,712 dual edges, 8 layers:
// 34.5 ms product by product, 5.48 ms here.  Per layer (cold L2): k_mlp_bwd 105 us
// (510 MB: 4.9 TB/s; one row a lane, whose 32-byte pieces lie in 32 lines an
// instruction, took 139), k_wgrad 94, k_reduce 70, k_edge_bwd 53 (4.8 TB/s),
// k_edge_dsum 144 once.
//
// Every mbarrier wait is bounded; one that gives up sets the error flag.
#include <utility>
#include <vector>

#include "fl_mpnn.cuh"

namespace fl {

__device__ __forceinline__ uint32_t positive_mask(uint32_t z) {  // 0xffff where a bf16 half is > 0
    const __nv_bfloat162 zero = __floats2bfloat162_rn(0.0f, 0.0f);
    return __hgt2_mask(*(const __nv_bfloat162 *)&z, zero);
}

// The 32 columns of row r (0: g, 1: g + 8) of a fragment (tmem_ld_frag32): the
// lane's eight consecutive ones from 8 q.
__device__ __forceinline__ void frag_to_row(const uint32_t (&v)[16], int r, int q, uint32_t (&x)[8]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        x[2 * j] = v[4 * j + 2 * r];
        x[2 * j + 1] = v[4 * j + 2 * r + 1];
    }
    transpose4(x[0], x[2], x[4], x[6], q);
    transpose4(x[1], x[3], x[5], x[7], q);
}

// Eight consecutive 16-bit values of row r to the packed fragment (tmem_st_frag_pairs).
__device__ __forceinline__ void pairs_to_frag(uint4 y, int r, int q, uint32_t (&w)[8]) {
    transpose4(y.x, y.y, y.z, y.w, q);
    w[r] = y.x;
    w[2 + r] = y.y;
    w[4 + r] = y.z;
    w[6 + r] = y.w;
}

// ------------------------------------------------------------- MLP backward
constexpr int MB_WARPS = 16, MB_THREADS = 32 * (MB_WARPS + 1);
constexpr int MB_CHUNKS = 8;
constexpr int MB_SMEM = MB_CHUNKS * MM_CHUNK_BYTES + 256 + 1024;

struct MlpBwdArgs {
    const float *dy;               // [M, ldy >= n2] fp32, or nullptr with dyb
    int64_t ldy;
    const __nv_bfloat16 *dyb;      // [M, 128] bf16 (n2 = 128): already rounded
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
    // the fp32 values that the bias gradients sum, [M, 128] each
    float *dz1f;                   // masked dz1
    float *daggf, *gf;             // message gradient x incoming edges; dagg W_e2 before the masks (layer)
    uint32_t *bits;                // [E, 4] which of an edge's 128 hidden activations are positive (layer)
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
                   d3 = in1 + 48, drain = in1 + 56, wbar = in1 + 64;
    uint32_t *tmem_slot = (uint32_t *)(bars + 9);
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
        mbar_init(wbar, MB_THREADS);
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
    fence_async_smem();
    tmem_fence_before();
    __syncthreads();
    cp_async_arrive_noinc(wbar);  // only the MMA warp waits for the weights
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
        bad = !warp_wait(wbar, 0);
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
        // lane = rows gq + 8 i (i < 4) of its warp's 32, 32 of the 128 columns;
        // in memory eight consecutive ones from 8 fq, so that four lanes cover
        // a row's whole 128-byte line
        const int quad = warp & 3, col = (warp >> 2) * 32, gq = lane >> 2, fq = lane & 3, mine = col + 8 * fq;
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16), operand = lanes + 384u + (uint32_t)(col / 2);
        auto hand_over = [&](uint32_t bar) {  // this warp's operand columns are written
            tmem_wait_st();
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        auto pack_row = [](const uint32_t (&x)[8]) {
            return make_uint4(pack_bf16x2(__uint_as_float(x[0]), __uint_as_float(x[1])),
                              pack_bf16x2(__uint_as_float(x[2]), __uint_as_float(x[3])),
                              pack_bf16x2(__uint_as_float(x[4]), __uint_as_float(x[5])),
                              pack_bf16x2(__uint_as_float(x[6]), __uint_as_float(x[7])));
        };
        int i = 0;
        for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x, ++i) {
            const int r0 = t * MM_BM + quad * 32 + gq;
            auto in = [&](int k) { return r0 + 8 * k < g.M; };
            auto at = [&](int k) { return (int64_t)(r0 + 8 * k) * MF_H + mine; };
            int rs[4], deg[4];
            if (MODE == 2) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    rs[k] = deg[k] = 0;
                    if (in(k)) {
                        rs[k] = g.start[r0 + 8 * k];
                        deg[k] = g.start[r0 + 8 * k + 1] - rs[k];
                    }
                }
            }
            // dy -> bf16
            if (col < g.n2) {  // (uniform over the warp)
                uint4 y[4];
                if (g.dy) {
                    float x[4][8];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
#pragma unroll
                        for (int u = 0; u < 8; ++u) x[k][u] = 0.0f;
                        if (in(k)) ld8f(g.dy + (int64_t)(r0 + 8 * k) * g.ldy + mine, x[k]);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        y[k] = make_uint4(pack_bf16x2(x[k][0], x[k][1]), pack_bf16x2(x[k][2], x[k][3]),
                                          pack_bf16x2(x[k][4], x[k][5]), pack_bf16x2(x[k][6], x[k][7]));
                        if (in(k)) *(uint4 *)(g.dz2 + (int64_t)(r0 + 8 * k) * g.n2 + mine) = y[k];
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        y[k] = make_uint4(0u, 0u, 0u, 0u);
                        if (in(k)) y[k] = *(const uint4 *)(g.dyb + at(k));
                    }
                }
                __syncwarp();
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t w[8];
#pragma unroll
                    for (int r = 0; r < 2; ++r) pairs_to_frag(y[2 * hh + r], r, fq, w);
                    tmem_st_frag_pairs(operand + ((uint32_t)(hh * 16) << 16), w);
                }
            }
            hand_over(in1);
            // dz1 = relu'(z) (dz2 W2)
            {
                uint4 z[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    z[k] = make_uint4(0u, 0u, 0u, 0u);
                    if (in(k)) z[k] = *(const uint4 *)(g.z + at(k));
                }
                __syncwarp();
                if (!warp_wait(d1, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const uint32_t half = (uint32_t)(hh * 16) << 16;
                    uint32_t v[16], m[8], w[8];
                    tmem_ld_frag32(lanes + half + (uint32_t)col, v);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const uint4 zz = z[2 * hh + r];
                        pairs_to_frag(make_uint4(positive_mask(zz.x), positive_mask(zz.y), positive_mask(zz.z), positive_mask(zz.w)),
                                      r, fq, m);
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j) {  // word j: columns 8 (j / 2) + 2 fq, + 1 of row j & 1
                        const int a = 4 * (j >> 1) + 2 * (j & 1);
                        v[a] = (m[j] & 0xffffu) ? v[a] : 0u;
                        v[a + 1] = (m[j] >> 16) ? v[a + 1] : 0u;
                        w[j] = pack_bf16x2(__uint_as_float(v[a]), __uint_as_float(v[a + 1]));
                    }
                    if (MODE > 0) tmem_st_frag_pairs(operand + half, w);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        uint32_t x[8];
                        frag_to_row(v, r, fq, x);
                        if (in(2 * hh + r)) {
                            *(uint4 *)(g.dz1 + at(2 * hh + r)) = pack_row(x);
                            st8u(g.dz1f + at(2 * hh + r), x);
                        }
                        __syncwarp();
                    }
                }
            }
            if (MODE == 0) {
                tmem_fence_before();
                continue;
            }
            hand_over(in2);
            if (MODE == 2) {
                // the message gradient, rounded
                if (!warp_wait(d2a, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const uint32_t half = (uint32_t)(hh * 16) << 16;
                    uint32_t v[16], w[8];
                    tmem_ld_frag32(lanes + half + 128u + (uint32_t)col, v);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int a = 4 * (j >> 1) + 2 * (j & 1);
                        w[j] = pack_bf16x2(__uint_as_float(v[a]), __uint_as_float(v[a + 1]));
                    }
                    tmem_st_frag_pairs(operand + 64u + half, w);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int k = 2 * hh + r;
                        uint32_t x[8];
                        frag_to_row(v, r, fq, x);
                        if (in(k)) {
                            *(uint4 *)(g.dagg + at(k)) = pack_row(x);
#pragma unroll
                            for (int u = 0; u < 8; ++u) x[u] = __float_as_uint(__uint_as_float(x[u]) * (float)deg[k]);
                            st8u(g.daggf + at(k), x);
                        }
                        __syncwarp();
                    }
                }
                hand_over(in3);
            }
            // dx (a layer: on top of dy, the residual's share)
            {
                float o[4][8];
                if (MODE == 2) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (in(k)) ld8f(g.dy + (int64_t)(r0 + 8 * k) * g.ldy + mine, o[k]);
                    __syncwarp();
                }
                if (!warp_wait(d2b, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t v[16];
                    tmem_ld_frag32(lanes + ((uint32_t)(hh * 16) << 16) + 256u + (uint32_t)col, v);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int k = 2 * hh + r;
                        uint32_t x[8];
                        frag_to_row(v, r, fq, x);
                        if (in(k)) {
                            if (MODE == 2) {
#pragma unroll
                                for (int u = 0; u < 8; ++u) x[u] = __float_as_uint(o[k][u] + __uint_as_float(x[u]));
                            }
                            st8u(g.dx + at(k), x);
                        }
                        __syncwarp();
                    }
                }
            }
            if (MODE == 2) {
                // dz_e of the cell's edges
                uint4 z[2][3];  // all the hidden activations of two rows' edges in flight
                auto fetch = [&](int hh) {
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            z[r][k] = make_uint4(0u, 0u, 0u, 0u);
                            if (k < deg[2 * hh + r])
                                z[r][k] = *(const uint4 *)(g.z1e + (int64_t)(rs[2 * hh + r] + k) * MF_H + mine);
                        }
                    __syncwarp();
                };
                fetch(0);
                if (!warp_wait(d3, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t v[16];
                    tmem_ld_frag32(lanes + ((uint32_t)(hh * 16) << 16) + (uint32_t)col, v);
                    if (hh == 1) fetch(1);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int n = 2 * hh + r;
                        uint32_t x[8];
                        frag_to_row(v, r, fq, x);
                        const uint4 w = pack_row(x);
                        if (in(n)) st8u(g.gf + at(n), x);
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            const uint4 p = make_uint4(positive_mask(z[r][k].x), positive_mask(z[r][k].y),
                                                       positive_mask(z[r][k].z), positive_mask(z[r][k].w));
                            uint32_t bits = (p.x & 1u) | (p.x >> 31) << 1 | (p.y & 1u) << 2 | (p.y >> 31) << 3 |
                                            (p.z & 1u) << 4 | (p.z >> 31) << 5 | (p.w & 1u) << 6 | (p.w >> 31) << 7;
                            bits <<= 8 * fq;
                            bits |= __shfl_xor_sync(0xffffffffu, bits, 1);
                            bits |= __shfl_xor_sync(0xffffffffu, bits, 2);
                            if (k < deg[n]) {
                                const int64_t e = rs[n] + k;
                                if (fq == 0) g.bits[e * 4 + col / 32] = bits;
                                *(uint4 *)(g.dze + e * MF_H + mine) = make_uint4(p.x & w.x, p.y & w.y, p.z & w.z, p.w & w.w);
                            }
                        }
                        __syncwarp();
                    }
                }
            }
            tmem_fence_before();
        }
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    cp_async_wait_all();
    tmem_fence_before();
    __syncthreads();
    if (warp == MB_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ------------------------------------------------------------- edge input gradients
constexpr int EB_PROD = 2, EB_EPI = 16, EB_THREADS = 32 * (EB_PROD + 1 + EB_EPI);
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

// Products p = 0..2: incoming slots, 3..5: outgoing slots of 128 cells; four
// 128-column TMEM regions in turn.
__global__ void __launch_bounds__(EB_THREADS, 1) k_edge_bwd(const __grid_constant__ EdgeBwdArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sW = smem_addr(smem), sR = sW + 4 * MM_CHUNK_BYTES;
    uint64_t *bars = (uint64_t *)(smem + (4 + EB_RING) * MM_CHUNK_BYTES);
    const uint32_t ringf = smem_addr(bars), ringe = ringf + 8 * EB_RING, df = ringe + 8 * EB_RING, de = df + 32, drain = de + 32, wbar = drain + 8;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * EB_RING + 4 + 4 + 2);
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
        mbar_init(wbar, EB_THREADS);
        mbar_fence_init();
    }
    if (warp == EB_PROD) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    for (int c = 0; c < 4; ++c)  // chunk = 64 K columns of 128 rows: receiver part 0, 1, sender part 0, 1
        load_weight_chunk(g.w1t + (c >> 1) * MF_H * g.ldw1t, g.ldw1t, MF_H, c & 1, sW + c * MM_CHUNK_BYTES, tid, EB_THREADS);
    fence_async_smem();
    tmem_fence_before();
    __syncthreads();
    cp_async_arrive_noinc(wbar);  // only the MMA warp waits for the weights
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
                int row[2][8];
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    rows_of_lane(p < 3 ? (p < deg[j] ? rs[j] + p : -1) : ord[j][p < 3 ? 0 : p - 3], row[j], lane);
                if (p == 3) load_orders(nso, nsd, nord);
#pragma unroll 1
                for (int c = 0; c < 2; ++c, ++q) {
                    const int s = q % EB_RING, u = q / EB_RING;
                    if (u > 0 && !warp_wait(ringe + 8 * s, (u - 1) & 1)) {
                        bad = true;
                        break;
                    }
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        warp_copy_numbered(g.dze + c * 64, MF_H, row[j], sR + s * MM_CHUNK_BYTES, 2 * warp + j, lane);
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
        bad = !warp_wait(wbar, 0);
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
        // lane = rows gq + 8 i of its warp's 32, 32 of the 128 columns
        const int quad = warp & 3, col = ((warp - EB_PROD - 1) >> 2) * 32, gq = lane >> 2, fq = lane & 3;
        const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)col;
        int m = 0;
        for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x) {
            const int c0 = t * MM_BM + quad * 32 + gq;
            float *row = g.dh + (int64_t)c0 * MF_H + col + 8 * fq;
            int deg[4];           // incoming edges, outgoing ones << 16
            float acc[32];        // [i][j][2], fragment order
            uint32_t tot[4][8];   // the rows' eight columns from 8 fq
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                deg[k] = 0;
                if (c0 + 8 * k < g.C) {
                    const int c = c0 + 8 * k;
                    deg[k] = (g.start[c + 1] - g.start[c]) | (g.send_start[c + 1] - g.send_start[c]) << 16;
                    ld8u(row + 8 * k * MF_H, tot[k]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int p = 0; p < 6; ++p, ++m) {
                if (!warp_wait(df + 8 * (m & 3), (m >> 2) & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t v[16];
                    tmem_ld_frag32(base + ((uint32_t)(hh * 16) << 16) + 128u * (m & 3), v);
                    if (hh == 1) {
                        tmem_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(de + 8 * (m & 3));
                    }
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int k = 2 * hh + r;
                        const bool valid = p < 3 ? p < (deg[k] & 0xffff) : p - 3 < (deg[k] >> 16);
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const float a = (p == 0 || p == 3) ? 0.0f : acc[8 * k + u];
                            acc[8 * k + u] = valid ? a + __uint_as_float(v[4 * (u >> 1) + 2 * r + (u & 1)]) : a;
                        }
                        if (p == 2 || p == 5) {
                            uint32_t x[8];
#pragma unroll
                            for (int u = 0; u < 8; ++u) x[u] = __float_as_uint(acc[8 * k + u]);
                            transpose4(x[0], x[2], x[4], x[6], fq);
                            transpose4(x[1], x[3], x[5], x[7], fq);
#pragma unroll
                            for (int u = 0; u < 8; ++u)
                                tot[k][u] = __float_as_uint(__uint_as_float(x[u]) + __uint_as_float(tot[k][u]));
                        }
                    }
                }
            }
            if (bad) break;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (c0 + 8 * k < g.C) st8u(row + 8 * k * MF_H, tot[k]);
            __syncwarp();
        }
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    cp_async_wait_all();
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
    float *outf;                               // the same before rounding (for the bias gradient)
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
                    const int r0 = t * 2 * MM_BM + j * MM_BM + 64 * warp;
                    warp_copy_span<64>(z, MF_H, r0, g.E, dst + j * MM_CHUNK_BYTES, 64 * warp, lane);
                }
                warp_copy_span<64>(w, g.ldwt[c >> 1], 64 * warp, MM_BN, dst + 2 * MM_CHUNK_BYTES, 64 * warp, lane);
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
                    float *f = g.outf + (int64_t)r * MF_H + half * 64 + hh * 32;
#pragma unroll
                    for (int u = 0; u < 32; u += 8) st8f(f + u, acc[hh] + u);
                }
                __syncwarp();
            }
        }
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    tmem_fence_before();
    __syncthreads();
    if (warp == ES_PROD) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ------------------------------------------------------------- weight gradients
constexpr int WG_PROD = 8, WG_EPI = 4, WG_THREADS = 32 * (WG_PROD + 1 + WG_EPI), WG_JOBS = 4;
constexpr int WG_BLOCK = 64 * 128;                  // 64 rows x 64 columns of bf16
constexpr int WG_RING_BYTES = 224 * 1024, WG_MAX_RING = 7;
constexpr int WG_SMEM = WG_RING_BYTES + 256 + 1024;
constexpr int WG_SPLITS = 512, WG_CTAS = 256;

struct WgSeg {
    const __nv_bfloat16 *base;
    const int32_t *rows;
    int64_t ld;
    int32_t width;                                  // 64 or 128
};

struct WgJob {
    WgSeg a, x[3];                                  // dZ (64 or 128 columns) and the segments of X
    int32_t nx, n_in, M;
    int32_t per, splits;                            // 64-row chunks per split, splits
    float *part;                                    // [splits, a.width, n_in]
};

// CTA b takes items first[b] .. first[b + 1] - 1: job << 14 | split.
struct WgArgs {
    WgJob job[WG_JOBS];
    int32_t *error;
    uint16_t first[WG_CTAS + 1];
    uint16_t item[WG_JOBS * WG_SPLITS];
};

// Splits of a product over M rows with n_in input features, those of the separate
// products (the same partial sums, so the same bits): at most 512, and at most 4 x 152
// accumulator tiles in all, a constant, so that the sums do not depend on the device.
// A split's length grows with the rows beyond that: 24 chunks (96 tensor-core steps)
// at 299,712 rows and 384 features, 440 at 5.7 M.
static void wg_split(int M, int n_in, int *per, int *splits) {
    const int chunks = (M + 63) / 64, tiles = (n_in + 127) / 128;
    const int want = std::max(1, std::min(std::min(chunks, WG_SPLITS), 4 * 152 / tiles));
    *per = (chunks + want - 1) / want;
    *splits = (chunks + *per - 1) / *per;
}

// Stage: 64 rows of dZ (two 64-column blocks of 8 KB) then of X's segments; as
// many as fit, so the ring is laid out anew where a CTA goes on to another job.
// Accumulators: columns 0 and 256 in turn for n_in <= 256, else both at once.
// Each split's accumulator is drained by the epilogue warps to its own slot.
__global__ void __launch_bounds__(WG_THREADS, 1) k_wgrad(const __grid_constant__ WgArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sR = smem_addr(smem);
    uint64_t *bars = (uint64_t *)(smem + WG_RING_BYTES);
    const uint32_t ringf = smem_addr(bars), ringe = ringf + 8 * WG_MAX_RING, accf = ringe + 8 * WG_MAX_RING, acce = accf + 16,
                   drain = acce + 16;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * WG_MAX_RING + 5);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int it0 = g.first[blockIdx.x], it1 = g.first[blockIdx.x + 1];
    if (tid == 0) {
        for (int s = 0; s < WG_MAX_RING; ++s) {
            mbar_init(ringf + 8 * s, 32 * WG_PROD);
            mbar_init(ringe + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(accf + 8 * b, 1);
            mbar_init(acce + 8 * b, WG_EPI);
        }
        mbar_init(drain, 1);
        mbar_fence_init();
    }
    if (warp == WG_PROD) {
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

    if (warp < WG_PROD) {
        // producers: 8 rows of each 64-row chunk, a lane rows own and own + 4;
        // row maps are read one chunk ahead.  The job's fields are held in
        // registers: read from the parameters in the copy loop they made it
        // 230 cycles an instruction
        uint32_t busy = 0u, par = 0u;  // per stage: filled and not known empty; parity of its next "empty"
        const int piece = lane & 7, own = 8 * warp + (lane >> 3);
        int s = 0, last = -1;
        for (int it = it0; it < it1 && !bad; ++it) {
            const int jn = g.item[it] >> 14, sp = g.item[it] & 0x3fff;
            const WgJob &J = g.job[jn];
            const int n_in = J.n_in, nx = J.nx, M = J.M, stage = (2 + n_in / 64) * WG_BLOCK;
            const int S = min(WG_MAX_RING, WG_RING_BYTES / stage);
            const WgSeg G[4] = {J.a, J.x[0], J.x[1], J.x[2]};
            if (jn != last) {  // another layout: every stage of the old one must be empty
                for (int k = 0; k < WG_MAX_RING && !bad; ++k) {
                    if (!(busy >> k & 1u)) continue;
                    if (!warp_wait(ringe + 8 * k, par >> k & 1u)) bad = true;
                    par ^= 1u << k;
                }
                if (bad) break;
                busy = 0u;
                s = 0;
                last = jn;
            }
            uint32_t off[4];
            off[0] = 0;
            off[1] = 2 * WG_BLOCK;
            off[2] = off[1] + (G[1].width / 64) * WG_BLOCK;
            off[3] = off[2] + (G[2].width / 64) * WG_BLOCK;
            const int c0 = sp * J.per, c1 = min((M + 63) / 64, c0 + J.per);
            auto load_rows = [&](int c, int (&o)[4][2]) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int r = c * 64 + own + 4 * i;
                    const bool in = c < c1 && r < M;
#pragma unroll
                    for (int x = 0; x < 4; ++x) o[x][i] = in && x <= nx ? (G[x].rows ? G[x].rows[r] : r) : -1;
                }
            };
            int row[4][2], nrow[4][2];
            load_rows(c0, row);
            for (int c = c0; c < c1; ++c) {
                load_rows(c + 1, nrow);
                if (busy >> s & 1u) {
                    if (!warp_wait(ringe + 8 * s, par >> s & 1u)) {
                        bad = true;
                        break;
                    }
                    par ^= 1u << s;
                }
                busy |= 1u << s;
                const uint32_t dst = sR + s * stage;
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    if (x <= nx) {
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int R = own + 4 * i;
                            const __nv_bfloat16 *src = row[x][i] >= 0 ? G[x].base + row[x][i] * G[x].ld : nullptr;
                            const uint32_t d = dst + off[x] + (uint32_t)(R * 128 + ((piece ^ (R & 7)) << 4));
                            if (src) cp_async16(d, src + piece * 8);
                            else asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(d), "r"(0u) : "memory");
                            // the upper 64 columns; dZ of 64: zero operand columns
                            if (src && G[x].width == 128) cp_async16(d + WG_BLOCK, src + 64 + piece * 8);
                            else if (x == 0 || G[x].width == 128)
                                asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(d + WG_BLOCK), "r"(0u) : "memory");
                        }
                    }
                }
                cp_async_arrive_noinc(ringf + 8 * s);
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int i = 0; i < 2; ++i) row[x][i] = nrow[x][i];
                if (++s == S) s = 0;
            }
        }
        cp_async_wait_all();
    } else if (warp == WG_PROD) {
        const bool issuer = elect_one();
        uint32_t par = 0u, used = 0u, upar = 0u;  // stages' next "full" parity; accumulators in use and their parity
        int s = 0, last = -1, turn = 0;
        bool wide = false;
        auto free_acc = [&](int b) {
            if (!(used >> b & 1u)) return;
            if (!warp_wait(acce + 8 * b, upar >> b & 1u)) bad = true;
            upar ^= 1u << b;
            used &= ~(1u << b);
        };
        for (int it = it0; it < it1 && !bad; ++it) {
            const int jn = g.item[it] >> 14, sp = g.item[it] & 0x3fff;
            const WgJob &J = g.job[jn];
            const int n_in = J.n_in, stage = (2 + n_in / 64) * WG_BLOCK, S = min(WG_MAX_RING, WG_RING_BYTES / stage);
            const int chunks = min((J.M + 63) / 64, (sp + 1) * J.per) - sp * J.per;
            if (jn != last) {
                s = 0;
                last = jn;
            }
            // at most 256 columns an instruction: columns [0, w0) and [256, n_in)
            const int w0 = min(256, n_in);
            const uint32_t i0 = umma_idesc_bf16_mn(w0), i1 = umma_idesc_bf16_mn(n_in > 256 ? n_in - 256 : 64);
            if (wide || n_in > 256) free_acc(0);
            if (n_in > 256) free_acc(1);
            wide = n_in > 256;
            const int b = wide ? 0 : turn;
            turn = b ^ 1;
            free_acc(b);
            if (bad) break;
            used |= 1u << b;
            tmem_fence_after();
            const uint32_t d = tmem + 256u * b;
            uint32_t acc = 0u;
            for (int c = 0; c < chunks; ++c) {
                if (!warp_wait(ringf + 8 * s, par >> s & 1u)) {
                    bad = true;
                    break;
                }
                par ^= 1u << s;
                fence_async_smem();
                if (issuer) {
                    const uint32_t a0 = sR + s * stage, x0 = a0 + 2 * WG_BLOCK;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {  // 16 rows each
                        const uint64_t da = umma_desc_mn_sw128(a0 + k * 2048, WG_BLOCK);
                        umma_bf16(d, da, umma_desc_mn_sw128(x0 + k * 2048, WG_BLOCK), i0, acc);
                        if (n_in > 256) umma_bf16(d + 256u, da, umma_desc_mn_sw128(x0 + 4 * WG_BLOCK + k * 2048, WG_BLOCK), i1, acc);
                        acc = 1u;
                    }
                    umma_commit(ringe + 8 * s);
                }
                if (++s == S) s = 0;
            }
            if (bad) break;
            if (issuer) umma_commit(accf + 8 * b);
        }
        if (issuer) umma_commit(drain);
        (void)warp_wait(drain, 0);
    } else {
        // epilogue: a warp's 32 output rows, 32 columns at a time in the fragment
        // shape; after the transposes a row's 32 columns are one 128-byte line
        // (a row a lane wrote 32-byte pieces, and the next split's accumulator
        // waited for them)
        const int quad = warp & 3, gq = lane >> 2, fq = lane & 3;
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        uint32_t par = 0u;
        int turn = 0;
        for (int it = it0; it < it1 && !bad; ++it) {
            const WgJob &J = g.job[g.item[it] >> 14];
            const int sp = g.item[it] & 0x3fff, n_in = J.n_in, rows = J.a.width;
            const int b = n_in > 256 ? 0 : turn;
            turn = b ^ 1;
            if (!warp_wait(accf + 8 * b, par >> b & 1u)) {
                bad = true;
                break;
            }
            par ^= 1u << b;
            tmem_fence_after();
            float *out = J.part + (int64_t)sp * rows * n_in + 8 * fq;
            for (int cb = 0; cb < n_in; cb += 32) {
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t v[16];
                    tmem_ld_frag32(lanes + ((uint32_t)(hh * 16) << 16) + 256u * b + (uint32_t)cb, v);
                    if (hh == 1 && cb + 32 >= n_in) {
                        tmem_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(acce + 8 * b);
                    }
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        uint32_t x[8];
                        frag_to_row(v, r, fq, x);
                        const int row = quad * 32 + gq + 8 * (2 * hh + r);
                        if (row < rows) st8u(out + (int64_t)row * n_in + cb, x);
                        __syncwarp();
                    }
                }
            }
        }
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    tmem_fence_before();
    __syncthreads();
    if (warp == WG_PROD) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ------------------------------------------------------------- sums over rows
constexpr int RD_JOBS = 4, RD_STRIDE = 256, CS_JOBS = 3, BF_JOBS = 112;

struct RdJob {
    const float *part;  // [count, n]
    float *out;         // [n], added to
    int32_t count, n;   // n a multiple of 4
};

// Column sums of x over M rows by row class (r mod 256): part[class][n].  With
// bits: row r counts x[map[r]] in the columns whose bit is set (a cell's
// message gradient over its edges).
struct CsJob {
    const float *x;
    const uint32_t *bits;    // [M, 4] or nullptr
    const int32_t *map;
    float *part;             // [256, n]
    int64_t ld;
    int32_t M, n;
};

struct RdArgs {
    RdJob job[RD_JOBS];
    CsJob cs[CS_JOBS];
    int32_t jobs, first;     // blockIdx.y: the first column sums, the partial products, the other column sums
};

struct BfJob {
    const float *part;       // [256, n]
    float *out;              // [n], added to
    int32_t n;
};

struct BfArgs {
    BfJob job[BF_JOBS];
};

__device__ __forceinline__ void add4(float4 &s, const float4 v) {
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
}

// Partial weight gradients: part[p] and part[p + 256], then over p in order.
// Column sums for the bias gradients: a thread per row class and column walks
// its rows in order (a sum's order is kept, so loads in flight, not adders,
// hide the latency: 16 rows by four columns a thread took 300 us a layer on
// 299,712 rows, 32 rows by one 80, of which the next batch's loads now overlap
// the adds).  Both in one launch: either alone leaves the device half idle.
__global__ void __launch_bounds__(256) k_reduce(const __grid_constant__ RdArgs g) {
    pdl_wait();
    pdl_launch_dependents();
    const int y = (int)blockIdx.y - g.first;
    if (y >= 0 && y < g.jobs) {
        const RdJob &J = g.job[y];
        const int n = J.n, count = J.count;
        const int i = ((int)blockIdx.x * 256 + (int)threadIdx.x) * 4;
        if (i >= n) return;
        float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float *p = J.part + i;
        const int lim = min(count, RD_STRIDE);
        for (int b = 0; b < lim; b += 8) {
            float4 v[8], w[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                v[u] = w[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (b + u < lim) v[u] = *(const float4 *)(p + (int64_t)(b + u) * n);
                if (b + u + RD_STRIDE < count) w[u] = *(const float4 *)(p + (int64_t)(b + u + RD_STRIDE) * n);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (b + u + RD_STRIDE < count) add4(v[u], w[u]);
                if (b + u < lim) add4(s, v[u]);
            }
        }
        float4 *o = (float4 *)(J.out + i);
        float4 v = *o;
        add4(v, s);
        *o = v;
        return;
    }
    // a thread per (row class, column): 32 columns a warp, 32 rows' loads in flight
    const CsJob &J = g.cs[y < 0 ? y + g.first : y - g.jobs + g.first];
    const int id = (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int cls = id >> 2, c = (id & 3) * 32 + lane, M = J.M;
    if (cls >= RD_STRIDE || (id & 3) * 32 >= J.n) return;  // (uniform over the warp)
    const float *x = J.x + c;
    const int64_t ld = J.ld;
    constexpr int N = 32, STEP = N * RD_STRIDE;  // rows of a batch; two batches' loads in flight
    float s = 0.0f, v[N], w[N];
    if (!J.bits) {
        auto fetch = [&](int r, float (&o)[N]) {
#pragma unroll
            for (int u = 0; u < N; ++u) {
                o[u] = 0.0f;
                if (r + u * RD_STRIDE < M) o[u] = x[(int64_t)(r + u * RD_STRIDE) * ld];
            }
        };
        auto add = [&](const float (&o)[N]) {
#pragma unroll
            for (int u = 0; u < N; ++u) s += o[u];
        };
        fetch(cls, v);
        for (int r = cls; r < M; r += 2 * STEP) {
            fetch(r + STEP, w);
            add(v);
            if (r + STEP >= M) break;
            fetch(r + 2 * STEP, v);
            add(w);
        }
    } else {
        const uint32_t *bits = J.bits + (id & 3);
        const int32_t *map = J.map;
        // the map entries and bits of a batch at once, a row a lane; rows past
        // the end read row 0 and have no bits (branches around the loads made
        // them wait for one another)
        auto load = [&](int r, int &row, uint32_t &m) {
            r += lane * RD_STRIDE;
            row = 0;
            m = 0u;
            if (r < M) {
                row = map[r];
                m = bits[(int64_t)r * 4];
            }
        };
        auto fetch = [&](int at, float (&o)[N]) {
#pragma unroll
            for (int u = 0; u < N; ++u) o[u] = x[(int64_t)__shfl_sync(0xffffffffu, at, u) * ld];
        };
        auto add = [&](uint32_t mask, const float (&o)[N]) {
#pragma unroll
            for (int u = 0; u < N; ++u) s += __shfl_sync(0xffffffffu, mask, u) >> lane & 1u ? o[u] : 0.0f;
        };
        int a0, a1, a2;
        uint32_t m0, m1, m2;
        load(cls, a0, m0);
        load(cls + STEP, a1, m1);
        fetch(a0, v);
        for (int r = cls; r < M; r += 2 * STEP) {
            load(r + 2 * STEP, a2, m2);
            fetch(a1, w);
            add(m0, v);
            if (r + STEP >= M) break;
            a0 = a2;
            m0 = m2;
            load(r + 3 * STEP, a2, m2);
            fetch(a0, v);
            add(m1, w);
            a1 = a2;
            m1 = m2;
        }
    }
    J.part[(int64_t)cls * J.n + c] = s;
}

// Bias gradients: the 256 class sums in order, added.
__global__ void __launch_bounds__(128) k_bias_final(const __grid_constant__ BfArgs g) {
    pdl_wait();
    pdl_launch_dependents();
    const BfJob &J = g.job[blockIdx.x];
    const int c = threadIdx.x;
    if (c >= J.n) return;
    float s = 0.0f;
    for (int b = 0; b < RD_STRIDE; b += 32) {
        float v[32];
#pragma unroll
        for (int u = 0; u < 32; ++u) v[u] = J.part[(b + u) * J.n + c];
#pragma unroll
        for (int u = 0; u < 32; ++u) s += v[u];
    }
    J.out[c] += s;
}

// floats of scratch that fl_mpnn_backward needs: the weight gradients' partials
// of the launch that has most, and every bias gradient's 256 class sums.
static int64_t wg_floats(int M, int n_out, int n_in) {
    int per = 0, splits = 0;
    if (M < 1) return 0;
    wg_split(M, n_in, &per, &splits);
    return (int64_t)splits * n_out * n_in;
}

static int64_t partial_floats(int C, int E, int L) {
    const int H = MF_H;
    const int64_t layer = wg_floats(E, H, 3 * H) + wg_floats(E, H, H) + wg_floats(C, H, 2 * H) + wg_floats(C, H, H);
    const int64_t enc = wg_floats(C, H, H) + wg_floats(C, H, 64) + wg_floats(E, H, H) + wg_floats(E, H, 64);
    const int64_t dec = wg_floats(C, 64, H) + wg_floats(C, H, H);
    return std::max(std::max(L > 0 ? layer : 0, enc), dec);
}

static int64_t backward_scratch(int C, int E, int L) { return partial_floats(C, E, L) + (int64_t)(3 * L + 6) * RD_STRIDE * MF_H; }

static cudaError_t current_sms(int *dev, int *sms) {
    cudaError_t e = cudaGetDevice(dev);
    return e == cudaSuccess ? cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, *dev) : e;
}

}  // namespace fl

using namespace fl;

extern "C" {

FL_API int fl_mpnn_backward_scratch(int32_t cells, int32_t edges, int32_t layers, int64_t *floats) {
    if (!floats || cells < 1 || edges < 0 || layers < 0)
        return set_error(FL_E_INVALID, "fl_mpnn_backward_scratch: bad sizes or NULL output");
    *floats = backward_scratch(cells, edges, layers);
    return FL_OK;
}

FL_API int fl_mpnn_backward(const FlMpnnBackwardDesc *d, void *stream) {
    if (!d || d->cells < 1 || d->edges < 0 || d->layers < 0 || d->layers > ES_MAX_LAYERS)
        return set_error(FL_E_INVALID, "fl_mpnn_backward: bad sizes (at most %d layers)", ES_MAX_LAYERS);
    const int C = d->cells, E = d->edges, L = d->layers;
    if (!d->x || !d->dy || !d->recv_start || !d->zn || !d->zd || !d->h_bf || !d->dh[0] || !d->dh[1] || !d->dz2c || !d->dz1c ||
        !d->dyb || !d->dz1f || !d->scratch ||
        (L > 0 && (!d->edge || !d->node || !d->agg || !d->z1n || !d->z1e || !d->dze || !d->dagg || !d->daggf || !d->gf || !d->send_start)) ||
        (E > 0 && (!d->src || !d->dst || !d->send_order || !d->ef || !d->ze || !d->e || !d->dz2e || !d->ef32 || !d->bits)))
        return set_error(FL_E_INVALID, "fl_mpnn_backward: NULL pointer");
    if (d->ldx < 64 || d->ldx % 8 || d->lde < 64 || d->lde % 8 || d->ldy < 64 || d->ldy % 8)
        return set_error(FL_E_INVALID, "fl_mpnn_backward: leading dimensions must be multiples of 8 and at least 64");
    uintptr_t a16 = (uintptr_t)d->x | (uintptr_t)d->ef;
    uintptr_t a32 = (uintptr_t)d->dy | (uintptr_t)d->zn | (uintptr_t)d->ze | (uintptr_t)d->e | (uintptr_t)d->zd |
                    (uintptr_t)d->dh[0] | (uintptr_t)d->dh[1] | (uintptr_t)d->dz2c | (uintptr_t)d->dz1c | (uintptr_t)d->dagg |
                    (uintptr_t)d->dyb | (uintptr_t)d->dz2e | (uintptr_t)d->dz1f | (uintptr_t)d->gf | (uintptr_t)d->ef32 |
                    (uintptr_t)d->scratch;
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
        ok = ok && d->h_bf[l] && d->agg[l] && d->z1n[l] && d->daggf[l] && (E == 0 || (d->z1e[l] && d->dze[l]));
        a32 |= (uintptr_t)d->h_bf[l] | (uintptr_t)d->agg[l] | (uintptr_t)d->z1n[l] | (uintptr_t)d->z1e[l] | (uintptr_t)d->dze[l] |
               (uintptr_t)d->daggf[l];
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
    if (e == cudaSuccess && d->scratch_floats < backward_scratch(C, E, L))
        return set_error(FL_E_INVALID, "fl_mpnn_backward: scratch of %lld floats, %lld needed", (long long)d->scratch_floats,
                         (long long)backward_scratch(C, E, L));
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
    float *part = d->scratch, *classes = part + partial_floats(C, E, L);
    const int c_tiles = (C + MM_BM - 1) / MM_BM, e_tiles = (E + MM_BM - 1) / MM_BM;

    // the weight gradients of up to four products in one launch, then every
    // partial sum.  The items (splits) go to the CTAs largest first, each to
    // the CTA with least to stage so far; a launch's jobs have the same sizes
    // in every layer, so the assignment is made once per kind of launch
    RdArgs rd;
    BfArgs bf_args;
    int n_rd = 0, n_cs = 0, n_bf = 0, rd_blocks = 0;
    auto sums = [&](const float *x, int64_t ld, int M, int n, float *gb, const uint32_t *bits = nullptr,
                    const int32_t *map = nullptr) {
        if (M < 1) return;
        rd.cs[n_cs++] = CsJob{x, bits, map, classes, ld, M, n};
        bf_args.job[n_bf++] = BfJob{classes, gb, n};
        classes += RD_STRIDE * MF_H;
        rd_blocks = std::max(rd_blocks, RD_STRIDE * 4 / 8);
    };
    auto reduce = [&]() {
        if (e != cudaSuccess) return;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)rd_blocks, (unsigned)(n_rd + n_cs));
        cfg.blockDim = dim3(256);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        rd.jobs = n_rd;
        // the longest chains start first: sums of more than 16 batches of rows,
        // the partial products (up to 32 batches), then the short sums, which
        // fill in.  The order changes no result and little time: a layer of 99,904
        // cells 70 us, with the products first 80, with them last 78, but a whole pass
        // on 10,082 / 49,928 / 100,352 / 180,000 / 401,408 cells 1.33 / 2.86 / 4.56 /
        // 7.41 / 14.40 ms, with the products first 1.33 / 2.85 / 4.57 / 7.44 / 14.40,
        // with them last 1.28 / 2.84 / 4.61 / 7.41 / 14.39
        std::sort(rd.cs, rd.cs + n_cs, [](const CsJob &a, const CsJob &b) { return a.M > b.M; });
        rd.first = 0;
        while (rd.first < n_cs && rd.cs[rd.first].M > 16 * 32 * RD_STRIDE) ++rd.first;
        e = cudaLaunchKernelEx(&cfg, k_reduce, rd);
        ++launched;
        n_rd = n_cs = rd_blocks = 0;
    };
    WgArgs wg;
    wg.error = err;
    int n_wg = 0, ctas = 0;
    bool planned = false;
    float *wg_out[WG_JOBS];
    auto seg = [](const void *p, const int32_t *rows, int64_t ld, int width) { return WgSeg{(const bf *)p, rows, ld, width}; };
    auto product = [&](int M, WgSeg a, std::initializer_list<WgSeg> xs, float *gw) {
        if (M < 1) return;
        WgJob &J = wg.job[n_wg];
        J = WgJob{};
        J.a = a;
        J.M = M;
        for (const WgSeg &x : xs) {
            J.x[J.nx++] = x;
            J.n_in += x.width;
        }
        wg_split(M, J.n_in, &J.per, &J.splits);
        wg_out[n_wg++] = gw;
    };
    auto plan = [&]() {
        ctas = std::min(sms, WG_CTAS);
        std::vector<std::vector<uint16_t>> list(ctas);
        std::vector<std::pair<int64_t, int>> load(ctas);  // heap: least loaded first, then the lower CTA
        for (int b = 0; b < ctas; ++b) load[b] = {0, b};
        int order[WG_JOBS];
        auto cost = [&](int j) { return (int64_t)wg.job[j].per * (wg.job[j].a.width + wg.job[j].n_in) + wg.job[j].n_in; };
        for (int j = 0; j < n_wg; ++j) order[j] = j;
        std::sort(order, order + n_wg, [&](int x, int y) { return cost(x) != cost(y) ? cost(x) > cost(y) : x < y; });
        auto more = [](const std::pair<int64_t, int> &x, const std::pair<int64_t, int> &y) { return x > y; };
        for (int k = 0; k < n_wg; ++k) {
            const int j = order[k];
            for (int sp = 0; sp < wg.job[j].splits; ++sp) {
                std::pop_heap(load.begin(), load.end(), more);
                list[load.back().second].push_back((uint16_t)(j << 14 | sp));
                load.back().first += cost(j);
                std::push_heap(load.begin(), load.end(), more);
            }
        }
        int n = 0, used = 0;
        for (int b = 0; b < ctas; ++b) {
            if (list[b].empty()) continue;
            wg.first[used++] = (uint16_t)n;
            for (uint16_t x : list[b]) wg.item[n++] = x;
        }
        wg.first[used] = (uint16_t)n;
        ctas = used;
    };
    auto flush = [&]() {
        if (e != cudaSuccess) return;
        float *p = part;
        for (int j = 0; j < n_wg; ++j) {
            WgJob &J = wg.job[j];
            J.part = p;
            p += (int64_t)J.splits * J.a.width * J.n_in;
            rd.job[n_rd++] = RdJob{J.part, wg_out[j], J.splits, J.a.width * J.n_in};
            rd_blocks = std::max(rd_blocks, (J.a.width * J.n_in + 1023) / 1024);
        }
        if (!planned) plan();
        planned = true;
        e = launch_blocks(k_wgrad, wg, ctas, sms, WG_THREADS, WG_SMEM, launched > 0, st);
        ++launched;
        n_wg = 0;
        reduce();
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
        a.dz1f = d->dz1f;
        a.n2 = 64;
        a.M = C;
        mlp(k_mlp_bwd<1>, a, c_tiles);
        sums(d->dy, d->ldy, C, 64, d->dec[1].gb);
        sums(d->dz1f, MF_H, C, MF_H, d->dec[0].gb);
        product(C, seg(d->dyb, nullptr, 64, 64), {seg(d->zd, nullptr, MF_H, MF_H)}, d->dec[1].gw);
        product(C, seg(d->dz1c, nullptr, MF_H, MF_H), {seg(d->h_bf[L], nullptr, MF_H, MF_H)}, d->dec[0].gw);
        flush();
    }
    int cur = 0;
    planned = false;
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
        a.dz1f = d->dz1f;
        a.daggf = d->daggf[l];
        a.gf = d->gf;
        a.bits = (uint32_t *)d->bits;
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
        sums(d->dh[cur], MF_H, C, MF_H, n2.gb);
        sums(d->dz1f, MF_H, C, MF_H, n1.gb);
        sums(d->gf, MF_H, E, MF_H, e1.gb, (const uint32_t *)d->bits, d->dst);
        product(E, seg(d->dze[l], nullptr, MF_H, MF_H),
                {seg(d->h_bf[l], d->dst, MF_H, MF_H), seg(d->h_bf[l], d->src, MF_H, MF_H), seg(d->e, nullptr, MF_H, MF_H)}, e1.gw);
        product(E, seg(d->dagg, d->dst, MF_H, MF_H), {seg(d->z1e[l], nullptr, MF_H, MF_H)}, e2.gw);
        product(C, seg(d->dz1c, nullptr, MF_H, MF_H),
                {seg(d->h_bf[l], nullptr, MF_H, MF_H), seg(d->agg[l], nullptr, MF_H, MF_H)}, n1.gw);
        product(C, seg(d->dz2c, nullptr, MF_H, MF_H), {seg(d->z1n[l], nullptr, MF_H, MF_H)}, n2.gw);
        flush();
    }
    // encoders
    planned = false;
    {
        MlpBwdArgs a{};
        a.dy = d->dh[cur];
        a.ldy = MF_H;
        a.z = (const bf *)d->zn;
        a.w2t = (const bf *)d->enc_n[1].wt;
        a.ldw2t = d->enc_n[1].ldwt;
        a.dz2 = (bf *)d->dz2c;
        a.dz1 = (bf *)d->dz1c;
        a.dz1f = d->dz1f;
        a.n2 = MF_H;
        a.M = C;
        mlp(k_mlp_bwd<0>, a, c_tiles);
        sums(d->dh[cur], MF_H, C, MF_H, d->enc_n[1].gb);
        sums(d->dz1f, MF_H, C, MF_H, d->enc_n[0].gb);
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
            b.outf = d->ef32;
            b.layers = L;
            b.E = E;
            b.error = err;
            e = launch_blocks(k_edge_dsum, b, (E + 2 * MM_BM - 1) / (2 * MM_BM), sms, ES_THREADS, ES_SMEM, true, st);
            ++launched;
        }
        sums(d->ef32, MF_H, E, MF_H, d->enc_e[1].gb);
        reduce();  // (the fp32 buffer is used again)
        MlpBwdArgs a{};
        a.dyb = (const bf *)d->dz2e;
        a.z = (const bf *)d->ze;
        a.w2t = (const bf *)d->enc_e[1].wt;
        a.ldw2t = d->enc_e[1].ldwt;
        a.dz1 = (bf *)d->dze[0];  // (no longer needed)
        a.dz1f = d->ef32;
        a.n2 = MF_H;
        a.M = E;
        mlp(k_mlp_bwd<0>, a, e_tiles);
        sums(d->ef32, MF_H, E, MF_H, d->enc_e[0].gb);
        product(E, seg(d->dz2e, nullptr, MF_H, MF_H), {seg(d->ze, nullptr, MF_H, MF_H)}, d->enc_e[1].gw);
        product(E, seg(d->dze[0], nullptr, MF_H, MF_H), {seg(d->ef, nullptr, d->lde, 64)}, d->enc_e[0].gw);
    }
    flush();
    if (e == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)n_bf);
        cfg.blockDim = dim3(128);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, k_bias_final, bf_args);
        ++launched;
    }
    if (e != cudaSuccess) return set_error(FL_E_CUDA, "fl_mpnn_backward: %s", cudaGetErrorString(e));
    add_launches(launched);
    return FL_OK;
}

}  // extern "C"
