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
// launch per product, 11.0 ms here (k_edge_fwd: the SM's shared-memory pipe, which
// MMA operands and gathers share, is full); 20,402 cells 777 -> 230 us (a
// launch's fill and drain, one or two tiles a CTA).
//
// Both kernels are persistent and warp-specialised: four producer warps
// (cp.async gathers into 16 KB stages; two warps, each copy's row pointer
// shuffled to its lanes, took 11.9 ms and 297 us), one MMA lane, sixteen epilogue
// warps; weights stay in shared memory, and only the MMA
// warp waits for them.  The rounding points (bf16 activations, fp32
// accumulation in K order, fp32 sums in edge order)
// are those of the separate products, so both give the same bits.
//
// Every mbarrier wait is bounded; one that gives up sets the error flag.
#include "fl_mpnn.cuh"

namespace fl {

constexpr int MF_PROD_WARPS = 4, MF_EPI_WARPS = 16, MF_THREADS = 32 * (MF_PROD_WARPS + 1 + MF_EPI_WARPS);
constexpr int MF_CHUNKS = 14;  // 16 KB chunks of shared memory
constexpr int MF_SMEM = MF_CHUNKS * MM_CHUNK_BYTES + 256 /* barriers */ + 1024 /* alignment */;
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

// Epilogue: warp = 32 rows (its TMEM lanes) x 32 columns in the fragment shape,
// so a lane needs only eight of a layer's biases and holds them for the whole
// kernel (read per row and column from shared memory, a four-wavefront
// broadcast each, they took a third of the shared-memory pipe that the MMA
// operands and the gathers need).  Four lanes hold a row's 32 columns; a 4 x 4
// transpose gives each eight consecutive ones for full 128-byte lines.
struct FragBias {
    float2 b[4];  // columns 8 j + 2 q, + 1
};

__device__ __forceinline__ FragBias frag_bias(const float *p, int q, bool in) {
    FragBias f;
#pragma unroll
    for (int j = 0; j < 4; ++j) f.b[j] = in ? make_float2(p[8 * j + 2 * q], p[8 * j + 2 * q + 1]) : make_float2(0.0f, 0.0f);
    return f;
}

// relu(v + bias) of 16 rows as bf16 pairs.
__device__ __forceinline__ void relu_pack_frag(const uint32_t (&v)[16], const FragBias &f, uint32_t (&w)[8]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
            w[2 * j + r] = pack_bf16x2(fmaxf(__uint_as_float(v[4 * j + 2 * r]) + f.b[j].x, 0.0f),
                                       fmaxf(__uint_as_float(v[4 * j + 2 * r + 1]) + f.b[j].y, 0.0f));
    }
}

// Row r (0: g, 1: g + 8) of packed pairs to global memory: 16 bytes a lane.
__device__ __forceinline__ void store_pairs(const uint32_t (&w)[8], int r, int q, __nv_bfloat16 *row, bool in) {
    uint32_t x0 = w[r], x1 = w[2 + r], x2 = w[4 + r], x3 = w[6 + r];
    transpose4(x0, x1, x2, x3, q);
    if (in) *(uint4 *)(row + 8 * q) = make_uint4(x0, x1, x2, x3);
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
    uint64_t *bars = (uint64_t *)(smem + MF_CHUNKS * MM_CHUNK_BYTES);
    const uint32_t dstf = smem_addr(bars), dste = dstf + 8, ringf = dstf + 16, ringe = ringf + 8 * EF_RING;
    const uint32_t d1f = ringe + 8 * EF_RING, zf = d1f + 24, d2f = zf + 16, de = d2f + 24, drain = de + 24, wbar = drain + 8;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 + 2 * EF_RING + 3 + 2 + 3 + 3 + 2);
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
        mbar_init(wbar, MF_THREADS);
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
    fence_async_smem();
    tmem_fence_before();
    __syncthreads();
    cp_async_arrive_noinc(wbar);  // only the MMA warp waits for the weights
    tmem_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool bad = false;
    pdl_wait();  // the previous kernel's activations; only then may the next one start
    pdl_launch_dependents();

    if (warp < MF_PROD_WARPS) {
        // producers: lane = tile row 32 * warp + lane; first edge, edge count
        // and senders, the next tile's read one tile ahead
        int t = blockIdx.x, q = 0;
        int rs, deg, snd[3];
        auto load_starts = [&](int tt, int &a, int &b) {
            const int c = tt * MM_BM + 32 * warp + lane;
            a = b = 0;
            if (tt < tiles && c < g.C) {
                a = g.start[c];
                b = g.start[c + 1] - a;
            }
        };
        auto load_senders = [&](int a, int b, int (&o)[3]) {
#pragma unroll
            for (int k = 0; k < 3; ++k) o[k] = k < b ? g.src[a + k] : -1;
        };
        load_starts(t, rs, deg);
        load_senders(rs, deg, snd);
        for (int i = 0; t < tiles && !bad; ++i) {
            const int tn = t + gridDim.x;
            int nrs, ndeg, nsnd[3];
            load_starts(tn, nrs, ndeg);
            if (i > 0 && !warp_wait(dste, (i - 1) & 1)) {
                bad = true;
                break;
            }
            int row[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                row[x] = t * MM_BM + 32 * warp + 4 * x + (lane >> 3);
                if (row[x] >= g.C) row[x] = -1;
            }
            warp_copy_numbered(g.h, MF_H, row, sD, warp, lane);
            warp_copy_numbered(g.h + 64, MF_H, row, sD + MM_CHUNK_BYTES, warp, lane);
            cp_async_arrive_noinc(dstf);
            load_senders(nrs, ndeg, nsnd);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
#pragma unroll
                for (int j = 0; j < 4; ++j, ++q) {
                    const int s = q % EF_RING, u = q / EF_RING;
                    if (u > 0 && !warp_wait(ringe + 8 * s, (u - 1) & 1)) {
                        bad = true;
                        break;
                    }
                    if (j == 0) rows_of_lane(snd[k], row, lane);
                    if (j == 2) rows_of_lane(k < deg ? rs + k : -1, row, lane);
                    warp_copy_numbered((j < 2 ? g.h : g.e) + (j & 1) * 64, MF_H, row, sR + s * MM_CHUNK_BYTES, warp, lane);
                    cp_async_arrive_noinc(ringf + 8 * s);
                }
                if (bad) break;
            }
            t = tn;
            rs = nrs;
            deg = ndeg;
#pragma unroll
            for (int k = 0; k < 3; ++k) snd[k] = nsnd[k];
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
            bad = !warp_wait(wbar, 0);
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
        // epilogue: lane = rows g + 8 i (i < 4) of its warp's 32, 32 of the 128 columns
        const int quad = warp & 3, col = ((warp - MF_PROD_WARPS - 1) >> 2) * 32, gq = lane >> 2, fq = lane & 3;
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        const FragBias f1 = frag_bias(g.b1 + col, fq, true), f2 = frag_bias(g.b2 + col, fq, true);
        float acc[32];  // [i][j][2]
        int n = 0, pt = 0, pdeg[4];
        // the messages of slot m (region k) of tile tt: summed, and stored after the last
        auto sum_slot = [&](int m, int k, int tt, const int (&deg)[4]) {
            if (!warp_wait(d2f + 8 * k, (m / 3) & 1)) {
                bad = true;
                return;
            }
            tmem_fence_after();
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                uint32_t v[16];
                tmem_ld_frag32(lanes + ((uint32_t)(hh * 16) << 16) + (uint32_t)(k * 128 + col), v);
                if (hh == 1) {
                    tmem_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(de + 8 * k);
                }
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int i = 2 * hh + r;
                    const bool valid = k < deg[i];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            const float msg = __uint_as_float(v[4 * j + 2 * r + x]) + (x ? f2.b[j].y : f2.b[j].x);
                            const float a = k == 0 ? 0.0f : acc[8 * i + 2 * j + x];
                            acc[8 * i + 2 * j + x] = valid ? a + msg : a;
                        }
                    }
                }
            }
            if (k == 2) {
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t w[8];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int r = 0; r < 2; ++r)
                            w[2 * j + r] = pack_bf16x2(acc[8 * (2 * hh + r) + 2 * j], acc[8 * (2 * hh + r) + 2 * j + 1]);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int c = tt * MM_BM + quad * 32 + gq + 8 * (2 * hh + r);
                        store_pairs(w, r, fq, g.agg + (int64_t)c * MF_H + col, c < g.C);
                    }
                }
                __syncwarp();
            }
        };
        for (int t = blockIdx.x, i = 0; t < tiles && !bad; t += gridDim.x, ++i) {
            int rs[4], deg[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int c = t * MM_BM + quad * 32 + gq + 8 * x;
                rs[x] = deg[x] = 0;
                if (c < g.C) {
                    rs[x] = g.start[c];
                    deg[x] = g.start[c + 1] - rs[x];
                }
            }
#pragma unroll
            for (int k = 0; k < 3; ++k, ++n) {
                if (!warp_wait(d1f + 8 * k, i & 1)) {
                    bad = true;
                    break;
                }
                tmem_fence_after();
                const uint32_t z = lanes + 384u + 64u * (n & 1) + (uint32_t)(col / 2);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t v[16], w[8];
                    const uint32_t half = (uint32_t)(hh * 16) << 16;
                    tmem_ld_frag32(lanes + half + (uint32_t)(k * 128 + col), v);
                    relu_pack_frag(v, f1, w);
                    tmem_st_frag_pairs(z + half, w);
                    if (g.z1) {
#pragma unroll
                        for (int r = 0; r < 2; ++r)
                            store_pairs(w, r, fq, g.z1 + (int64_t)(rs[2 * hh + r] + k) * MF_H + col, k < deg[2 * hh + r]);
                        __syncwarp();
                    }
                }
                tmem_wait_st();
                tmem_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(zf + 8 * (n & 1));
                if (n > 0) {
                    if (k == 0) sum_slot(n - 1, 2, pt, pdeg);
                    else sum_slot(n - 1, k - 1, t, deg);
                }
                if (bad) break;
            }
            pt = t;
#pragma unroll
            for (int x = 0; x < 4; ++x) pdeg[x] = deg[x];
        }
        if (n > 0 && !bad) sum_slot(n - 1, 2, pt, pdeg);
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    cp_async_wait_all();
    tmem_fence_before();
    __syncthreads();
    if (warp == MF_PROD_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

__global__ void __launch_bounds__(MF_THREADS, 1) k_mlp2(const __grid_constant__ Mlp2Args g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int nK = g.nk[0] + g.nk[1], S = g.ring;
    const uint32_t sW1 = smem_addr(smem), sW2 = sW1 + nK * MM_CHUNK_BYTES, sR = sW2 + 2 * MM_CHUNK_BYTES;
    uint64_t *bars = (uint64_t *)(smem + MF_CHUNKS * MM_CHUNK_BYTES);
    const uint32_t ringf = smem_addr(bars), ringe = ringf + 8 * M2_MAX_RING;
    const uint32_t d1f = ringe + 8 * M2_MAX_RING, zf = d1f + 24, d2f = zf + 16, de = d2f + 24, drain = de + 24, wbar = drain + 8;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * M2_MAX_RING + 3 + 2 + 3 + 3 + 2);
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
        mbar_init(wbar, MF_THREADS);
        mbar_fence_init();
    }
    if (warp == MF_PROD_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    for (int c = 0; c < nK; ++c) load_weight_chunk(g.w1, g.ldw1, MF_H, c, sW1 + c * MM_CHUNK_BYTES, tid, MF_THREADS);
    for (int c = 0; c < 2; ++c) load_weight_chunk(g.w2, g.ldw2, g.n2, c, sW2 + c * MM_CHUNK_BYTES, tid, MF_THREADS);
    fence_async_smem();
    tmem_fence_before();
    __syncthreads();
    cp_async_arrive_noinc(wbar);  // only the MMA warp waits for the weights
    tmem_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool bad = false;
    pdl_wait();
    pdl_launch_dependents();

    if (warp < MF_PROD_WARPS) {
        int s = 0, u = 0;
        for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x) {
            int row[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                row[i] = t * MM_BM + 32 * warp + 4 * i + (lane >> 3);
                if (row[i] >= g.M) row[i] = -1;
            }
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                for (int c = 0; c < g.nk[x] && !bad; ++c) {
                    if (u > 0 && !warp_wait(ringe + 8 * s, (u - 1) & 1)) {
                        bad = true;
                        break;
                    }
                    warp_copy_numbered(g.a[x] + c * 64, g.lda[x], row, sR + s * MM_CHUNK_BYTES, warp, lane);
                    cp_async_arrive_noinc(ringf + 8 * s);
                    if (++s == S) {
                        s = 0;
                        ++u;
                    }
                }
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
            bad = !warp_wait(wbar, 0);
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
        // epilogue: lane = rows g + 8 i (i < 4) of its warp's 32, 32 of the 128 columns
        const int quad = warp & 3, col = ((warp - MF_PROD_WARPS - 1) >> 2) * 32, gq = lane >> 2, fq = lane & 3;
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        const bool has_out = col < g.n2;  // (n2 = 64: the upper columns do not exist)
        const FragBias f1 = frag_bias(g.b1 + col, fq, true), f2 = frag_bias(g.b2 + col, fq, has_out);
        int n = 0, pt = 0;
        auto finish = [&](int m, int tt) {
            const int k = m % 3;
            // the residual's rows, eight consecutive columns a lane, on their way during the wait
            float res[4][8];
            const int64_t r0 = (int64_t)tt * MM_BM + quad * 32 + gq;
            if (g.residual && has_out) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (r0 + 8 * i < g.M) ld8f(g.residual + (r0 + 8 * i) * MF_H + col + 8 * fq, res[i]);
                __syncwarp();
            }
            if (!warp_wait(d2f + 8 * k, (m / 3) & 1)) {
                bad = true;
                return;
            }
            tmem_fence_after();
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                uint32_t v[16];
                tmem_ld_frag32(lanes + ((uint32_t)(hh * 16) << 16) + (uint32_t)(k * 128 + col), v);
                if (hh == 1) {
                    tmem_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(de + 8 * k);
                }
                if (!has_out) continue;  // (uniform over the warp)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int i = 2 * hh + r;
                    uint32_t x[8];  // columns 8 fq .. + 7 of the row after the transposes
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        x[2 * j] = __float_as_uint(__uint_as_float(v[4 * j + 2 * r]) + f2.b[j].x);
                        x[2 * j + 1] = __float_as_uint(__uint_as_float(v[4 * j + 2 * r + 1]) + f2.b[j].y);
                    }
                    transpose4(x[0], x[2], x[4], x[6], fq);
                    transpose4(x[1], x[3], x[5], x[7], fq);
                    const int64_t row = r0 + 8 * i;
                    if (row < g.M) {
                        float y[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) y[u] = __uint_as_float(x[u]);
                        if (g.residual) {
#pragma unroll
                            for (int u = 0; u < 8; ++u) y[u] += res[i][u];
                        }
                        const int64_t o = row * g.n2 + col + 8 * fq;
                        if (g.out_f32) st8f(g.out_f32 + o, y);
                        if (g.out_bf16)
                            *(uint4 *)(g.out_bf16 + o) = make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]),
                                                                    pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7]));
                    }
                    __syncwarp();
                }
            }
        };
        for (int t = blockIdx.x; t < tiles && !bad; t += gridDim.x, ++n) {
            const int k = n % 3;
            if (!warp_wait(d1f + 8 * k, (n / 3) & 1)) {
                bad = true;
                break;
            }
            tmem_fence_after();
            const uint32_t z = lanes + 384u + 64u * (n & 1) + (uint32_t)(col / 2);
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                uint32_t v[16], w[8];
                const uint32_t half = (uint32_t)(hh * 16) << 16;
                tmem_ld_frag32(lanes + half + (uint32_t)(k * 128 + col), v);
                relu_pack_frag(v, f1, w);
                tmem_st_frag_pairs(z + half, w);
                if (g.z1) {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int64_t row = (int64_t)t * MM_BM + quad * 32 + gq + 8 * (2 * hh + r);
                        store_pairs(w, r, fq, g.z1 + row * MF_H + col, row < g.M);
                    }
                    __syncwarp();
                }
            }
            tmem_wait_st();
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(zf + 8 * (n & 1));
            if (n > 0) finish(n - 1, pt);
            pt = t;
        }
        if (n > 0 && !bad) finish(n - 1, pt);
    }
    if (bad) atomicCAS(g.error, 0, FL_E_TIMEOUT);
    cp_async_wait_all();
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
