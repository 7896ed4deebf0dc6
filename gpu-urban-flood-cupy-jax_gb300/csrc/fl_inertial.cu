// Local-inertial surface step for sm_103a (solver.surface_step_mode =
// "local_inertial"): the reference's fast routing mode
// (gurugram_flood/kernels/triangular_local_inertial_cuda_kernels.py:59-262,
// triangular_backend.py:531-590, local_inertial.py:20-49) as two launches:
//   k_li_edges  one thread per edge: the LISFLOOD-style discharge update from
//               the water-surface slope (face distance and Manning n are
//               static per edge), written into the (cell, slot) place of
//               each of its cells                                   [:59-167]
//   k_li_cells  one thread per cell: the donor limit factors (a cell's volume
//               over the summed outgoing requests of its edges, in slot
//               order; the reference adds them with atomicAdd) of the cell
//               and of each neighbour that donates to it [:172-189], the
//               volume change, momentum from the face discharges, then the
//               same sources, clamp, external inflow, wet time and snapshots
//               as the full-SWE surface kernel; its last block plans the next
//               step                                                [:194-262]
// The cell kernel reads its cell's discharges and slot tables (flags, the
// other cell, the face normals) contiguously and gathers a donating
// neighbour's slots, depth and area.
//
//   k_li_tiles  the same step in one launch over tiles of 256 cells with their
//               two rings of neighbours in shared memory: the discharges of the
//               tile's and ring 1's edges, the donor factors of own and ring-1
//               cells, the own cells' update.  The two launches write every
//               discharge to memory and read it back through scattered slots
//               (186 MB a step on 981,880 cells, 67.3 us chained); here about a
//               quarter of the edges are evaluated a second time, beside another
//               tile, and no discharge leaves the SM: 33 us, of which the
//               compulsory 128 MB take 19 and the IEEE divisions and cube roots
//               of 1.9 M entries most of the rest.
//
// k_li_tiles runs where the rings of every tile fit its 10-bit local indices and
// shared memory (cells in space-filling-curve order do, 46 + 50 halo cells a
// tile); cells in an order of the caller's without centroids take the two launches.
// Compiled with -fmad=false: the discharge arithmetic is rounded as written.
#include <cuda_runtime.h>

#include "fl_device.cuh"
#include "fl_run.cuh"

namespace fl {

__global__ void __launch_bounds__(256) k_li_edges(const __grid_constant__ LiArgs a, int slot) {
    pdl_launch_dependents();  // the cell kernel may launch and wait meanwhile
    pdl_wait();               // the previous step's kernels
    const StepCtrl s = a.ctrl[slot];
    if (!s.active || !(s.phases & FL_PHASE_SURFACE)) return;
    const float4 *__restrict__ in = s.parity ? a.state1 : a.state0;
    const float dt = s.dt_f, g = a.g;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < a.E; e += gridDim.x * blockDim.x) {
        const int2 lr = a.e_lr[e];
        const float4 geo = a.e_geo[e];
        const uint32_t f = __float_as_uint(geo.w);
        const int L = lr.x, R = (f & LI_INTERIOR) ? lr.y : lr.x;
        const bool la = (f & LI_LACTIVE) != 0, ra = (f & LI_RACTIVE) != 0, ai = (f & LI_AI) != 0;
        const bool bedge = (f & LI_BEDGE) != 0;
        const float4 sl = in[L], sr = in[R];
        const float hl = la ? sl.x : 0.0f, hul = la ? sl.y : 0.0f, hvl = la ? sl.z : 0.0f;
        const float hr = ra ? sr.x : 0.0f, hur = ra ? sr.y : 0.0f, hvr = ra ? sr.z : 0.0f;
        const float bl = sl.w, br = sr.w;
        const float etal = bl + hl;
        const float etar = ai ? br + hr : bl;
        const float bstar = ai ? fmax32(bl, br) : bl;
        const float hflow = fmax32(fmax32(etal, etar) - bstar, 0.0f);
        const float2 dm = a.e_dm[e];  // {max(0.5 (l_L + l_R), 1e-6), face n}, formed on the host in float32
        const float slope = (etar - etal) / dm.x;
        const float nx = geo.x, ny = geo.y, len = geo.z;
        const float nl = hul * nx + hvl * ny, nr = hur * nx + hvr * ny;
        const float qold = (ai ? 0.5f * (nl + nr) : nl) * len;
        const float mn = dm.y;
        const float area = fmax32(hflow * len, 1.0e-8f);
        const float radius = fmax32(hflow, 1.0e-6f);
        const float r43 = radius * cbrtf(radius);
        const float numer = qold - g * area * dt * slope;
        const float fric = 1.0f + g * dt * mn * mn * fabsf(qold) / (r43 * area);
        float q = numer / fric;
        if (!(ai || bedge)) q = 0.0f;
        if (bedge) q = fmax32(q, 0.0f);
        float *qs = reinterpret_cast<float *>(a.Qs);
        qs[(size_t)L * 4 + ((f >> LI_SLOTL_SHIFT) & 3u)] = q;
        if (f & LI_INTERIOR) qs[(size_t)lr.y * 4 + ((f >> LI_SLOTR_SHIFT) & 3u)] = q;
    }
}

// Donor limit factor of a cell (reference :172-189): its volume over the
// summed outgoing requests of its active interior edges, in slot order (the
// reference adds them with atomicAdd).  sb, q4: the cell's slot bits and
// discharges; h, area: its depth at the step start and its area.  The cell
// kernel evaluates it for a cell and for each neighbour that donates to it;
// every evaluation of one cell reads the same values, so all agree
// bit-for-bit (this file is compiled without contraction).
__device__ __forceinline__ float li_donor_scale(uint32_t sb, float4 q4, float h, float area, float dt) {
    const float qk[3] = {q4.x, q4.y, q4.z};
    float req = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint32_t b = sb >> (4 * k);
        if (!(b & LIS_PRESENT) || !(b & LIS_AI)) continue;
        const float q = qk[k];
        if (q == 0.0f) continue;
        // the donor is the left cell for q >= 0, else the right one
        if ((q >= 0.0f) == ((b & LIS_LEFT) != 0)) req += fabsf(q) * dt;
    }
    const float vol = fmax32(h, 0.0f) * area;
    return req > 1.0e-12f ? fmin32(1.0f, vol / req) : 1.0f;
}

template <int KIND>
__global__ void __launch_bounds__(256) k_li_cells(const __grid_constant__ LiArgs a, int slot, int plan_next) {
    pdl_wait();  // the discharges of k_li_edges (and every earlier kernel's writes)
    if ((int)blockIdx.x == (int)gridDim.x - 1) {  // the last block plans the next step
        if (plan_next && threadIdx.x == 0) plan_step(a.run, a.snap_t, a.hy, &a.ctrl[slot ^ 1], false, 0.0f, FL_PHASE_ALL);
        return;
    }
    const StepCtrl s = a.ctrl[slot];
    if (!s.active) return;
    const float4 *__restrict__ in = s.parity ? a.state1 : a.state0;
    float4 *__restrict__ out = s.parity ? a.state0 : a.state1;
    const float dt = s.dt_f, md = a.md;
    const bool do_surface = (s.phases & FL_PHASE_SURFACE) != 0;
    const bool drain_finishes = (s.phases & FL_PHASE_DRAINAGE) != 0;
    const bool recharge_finishes = (s.phases & FL_PHASE_RECHARGE) != 0;
    float led[SURF_TERMS] = {0.0f, 0.0f, 0.0f, 0.0f};
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < a.C) {
        const float4 st = in[c];
        const float4 ci = a.cinfo[c];
        const uint32_t info = __float_as_uint(ci.z);
        if (s.check_finite && !isfinite(st.x)) {
            if (atomicCAS(&a.run->error, 0, FL_E_NONFINITE) == 0) a.run->error_step = s.step;
        }
        float wt = 0.0f;
        float4 hz = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
        if (KIND == 1) {
            wt = a.wet[c];
            hz = a.horton[c];
        }
        float hn = 0.0f, hun = 0.0f, hvn = 0.0f;
        if (!do_surface) {
            hn = st.x; hun = st.y; hvn = st.z;
        } else if (info & CELL_ACTIVE) {
            // the cell's face discharges in slot order
            const uint32_t sb = a.c_bits[c];
            const float4 q4 = a.Qs[c];
            const int4 oc = a.c_other[c];
            const float qk[3] = {q4.x, q4.y, q4.z};
            const int ok[3] = {oc.x, oc.y, oc.z};
            const float own_scale = li_donor_scale(sb, q4, st.x, ci.x, dt);
            float hd = 0.0f, qx = 0.0f, qy = 0.0f, bf = 0.0f;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const uint32_t b = sb >> (4 * k);
                if (!(b & LIS_PRESENT)) continue;
                const float q = qk[k];
                if (q == 0.0f) continue;
                const float2 nrm = a.c_nrm[(size_t)k * (size_t)a.C + (size_t)c];
                if (b & LIS_INTERIOR) {
                    const bool left = (b & LIS_LEFT) != 0;
                    float sd = own_scale;
                    if ((q >= 0.0f) != left) {  // the neighbour donates: its factor from its own slots
                        const int m = ok[k];
                        sd = li_donor_scale(a.c_bits[m], a.Qs[m], in[m].x, a.cinfo[m].x, dt);
                    }
                    const float lim = q * sd * dt;
                    hd += left ? -lim : lim;
                } else {
                    const float bq = q * dt;
                    hd -= bq;
                    bf += bq;
                }
                qx += q * nrm.x;
                qy += q * nrm.y;
            }
            const float area = ci.x;
            const float h0 = fmax32(st.x + hd / area, 0.0f);
            const float per = 2.0f * area / fmax32(a.char_len[c], 1.0e-12f);
            const bool wet0 = h0 > md;
            const float hu0 = wet0 ? qx / fmax32(per, 1.0e-12f) : 0.0f;
            const float hv0 = wet0 ? qy / fmax32(per, 1.0e-12f) : 0.0f;
            // _apply_sources (reference triangular_backend.py:1330-1379)
            const float rain = KIND == 1 ? s.rain_f * hz.w : s.rain_f;
            const float infil = KIND == 1 ? hz.y + (hz.x - hz.y) * __expf(-hz.z * wt) : a.infil_scalar;
            const float rd = fmax32(rain, 0.0f) * dt;
            const float h1 = h0 + rd;
            const float id = fmin32(h1, fmax32(infil, 0.0f) * dt);
            const float h2 = h1 - id;
            const float sc = (h1 > md) ? h2 / fmax32(h1, md) : 0.0f;
            const bool wet2 = h2 > md;
            hn = h2;
            hun = wet2 ? hu0 * sc : 0.0f;
            hvn = wet2 ? hv0 * sc : 0.0f;
            led[0] += rd * area;
            led[1] += id * area;
            led[3] += bf;
        }
        if (s.phases & FL_PHASE_CLAMP) clamp_velocity_exact(hn, hun, hvn, a.vmax);
        if ((info & CELL_RECEIVER) && (s.phases & FL_PHASE_INFLOW)) hn = __fadd_rn(hn, a.ext_add[c]);
        out[c] = make_float4(hn, hun, hvn, st.w);
        const bool final_here = !(drain_finishes && (info & CELL_COUPLED)) &&
                                !(recharge_finishes && (info & CELL_RECHARGE));
        if (KIND == 1 && do_surface && final_here) a.wet[c] = wt + dt * (float)(hn > md);
        if (s.snap_slot >= 0) {
            const size_t o = (size_t)s.snap_slot * (size_t)a.C + (size_t)c;
            if (final_here) a.snap_h[o] = hn;
            a.snap_hu[o] = hun;
            a.snap_hv[o] = hvn;
        }
    }
    warp_add_ledger<SURF_TERMS>(led, a.ledger);
}

constexpr uint64_t LT_WAIT_NS = 1000000000ull;  // 1 s per wait on a tile copy

struct LtStage {
    float4 *st, *ci, *hz, *en;
    float *wt, *cl, *ha;
    float2 *dm;
    int32_t *hs;
};

__device__ __forceinline__ LtStage lt_stage(const LiTileArgs &a, unsigned char *smem, int s) {
    unsigned char *b = smem + a.off_stage + s * a.stage_bytes;
    LtStage t;
    t.st = (float4 *)b;
    t.ci = (float4 *)(b + a.so_ci);
    t.hz = (float4 *)(b + a.so_hz);
    t.wt = (float *)(b + a.so_wt);
    t.cl = (float *)(b + a.so_cl);
    t.en = (float4 *)(b + a.so_en);
    t.dm = (float2 *)(b + a.so_dm);
    t.hs = (int32_t *)(b + a.so_hs);
    t.ha = (float *)(b + a.so_ha);
    return t;
}

// Bytes of a tile's static copies, and of those of what a step writes (exactly
// the copies that lt_issue_static and lt_issue_step make).
template <int KIND>
__device__ __forceinline__ uint32_t lt_static_bytes(const int4 ti, const int4 tj) {
    return TILE * 16u + (KIND == 1 ? TILE * 16u : 0u) + TILE * 4u + (uint32_t)ti.y * 24u + (uint32_t)((ti.w + 3) & ~3) * 4u +
           (uint32_t)((tj.x + 3) & ~3) * 4u;
}
template <int KIND>
__device__ __forceinline__ uint32_t lt_step_bytes() {
    return TILE * 16u + (KIND == 1 ? TILE * 4u : 0u);
}

template <int KIND>
__device__ __forceinline__ void lt_issue_static(const LiTileArgs &a, const LtStage &S, const int4 ti, const int4 tj, uint32_t bar,
                                                int t) {
    const size_t c0 = (size_t)t * TILE;
    bulk_copy_g2s(smem_addr(S.ci), a.c.cinfo + c0, TILE * 16u, bar);
    bulk_copy_g2s(smem_addr(S.cl), a.char_len + c0, TILE * 4u, bar);
    if (KIND == 1) bulk_copy_g2s(smem_addr(S.hz), a.c.horton + c0, TILE * 16u, bar);
    const uint32_t hb = (uint32_t)((ti.w + 3) & ~3) * 4u, ab = (uint32_t)((tj.x + 3) & ~3) * 4u;
    if (ti.y) {
        bulk_copy_g2s(smem_addr(S.en), a.ent + ti.x, (uint32_t)ti.y * 16u, bar);
        bulk_copy_g2s(smem_addr(S.dm), a.dm + ti.x, (uint32_t)ti.y * 8u, bar);
    }
    if (hb) bulk_copy_g2s(smem_addr(S.hs), a.halo_src + ti.z, hb, bar);
    if (ab) bulk_copy_g2s(smem_addr(S.ha), a.harea + tj.y, ab, bar);
}

template <int KIND>
__device__ __forceinline__ void lt_issue_step(const float4 *in, const float *wet, const LtStage &S, uint32_t bar, int t) {
    const size_t c0 = (size_t)t * TILE;
    bulk_copy_g2s(smem_addr(S.st), in + c0, TILE * 16u, bar);
    if (KIND == 1) bulk_copy_g2s(smem_addr(S.wt), wet + c0, TILE * 4u, bar);
}

__device__ __forceinline__ void lt_sync() { asm volatile("bar.sync 1, %0;" ::"n"(TILE) : "memory"); }

__device__ __forceinline__ bool lt_all(bool p) {
    uint32_t r;
    asm volatile(
        "{\n"
        ".reg .pred pi, po;\n"
        "setp.ne.u32 pi, %1, 0;\n"
        "bar.red.and.pred po, 1, %2, pi;\n"
        "selp.u32 %0, 1, 0, po;\n"
        "}\n"
        : "=r"(r)
        : "r"((uint32_t)p), "n"(TILE)
        : "memory");
    return r != 0;
}

// One tile entry: the edge's discharge (k_li_edges' arithmetic) into the (cell,
// slot) places {q, q nx, q ny, slot bits | the other cell's index << 8}.
__device__ __forceinline__ void lt_entry(const float4 en, const float2 dm, const float4 *st, float4 *slots, float g, float dt) {
    const uint32_t f = __float_as_uint(en.w);
    const uint32_t L = (f >> LT_LEFT_SHIFT) & LT_IDX_MASK, Ri = (f >> LT_RIGHT_SHIFT) & LT_IDX_MASK;
    const bool ai = (f & LT_AI) != 0;
    const float4 sl = st[L], sr = st[ai ? Ri : L];
    const float bl = sl.w, br = sr.w;
    const float etal = bl + sl.x;
    const float etar = ai ? br + sr.x : bl;
    const float bstar = ai ? fmax32(bl, br) : bl;
    const float hflow = fmax32(fmax32(etal, etar) - bstar, 0.0f);
    const float slope = (etar - etal) / dm.x;
    const float nx = en.x, ny = en.y, len = en.z;
    const float nl = sl.y * nx + sl.z * ny, nr = sr.y * nx + sr.z * ny;
    const float qold = (ai ? 0.5f * (nl + nr) : nl) * len;
    const float mn = dm.y;
    const float area = fmax32(hflow * len, 1.0e-8f);
    const float radius = fmax32(hflow, 1.0e-6f);
    const float r43 = radius * cbrtf(radius);
    const float numer = qold - g * area * dt * slope;
    const float fric = 1.0f + g * dt * mn * mn * fabsf(qold) / (r43 * area);
    float q = numer / fric;
    if (!ai) q = fmax32(q, 0.0f);
    const float qx = q * nx, qy = q * ny;
    const uint32_t kind = LIS_PRESENT | (ai ? LIS_AI | LIS_INTERIOR : 0u);
    if (f & LT_LKEEP)
        slots[L * 3 + ((f >> LT_SLOTL_SHIFT) & 3u)] = make_float4(q, qx, qy, __uint_as_float(kind | LIS_LEFT | Ri << 8));
    if (f & LT_RKEEP) slots[Ri * 3 + ((f >> LT_SLOTR_SHIFT) & 3u)] = make_float4(q, qx, qy, __uint_as_float(kind | L << 8));
}

// li_donor_scale over a cell's places in shared memory.
__device__ __forceinline__ float lt_donor_scale(const float4 *slots, float h, float area, float dt) {
    float req = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 v = slots[k];
        const uint32_t b = __float_as_uint(v.w);
        if (!(b & LIS_AI) || v.x == 0.0f) continue;
        if ((v.x >= 0.0f) == ((b & LIS_LEFT) != 0)) req += fabsf(v.x) * dt;
    }
    const float vol = fmax32(h, 0.0f) * area;
    return req > 1.0e-12f ? fmin32(1.0f, vol / req) : 1.0f;
}

// An active own cell's update from its places and the donor factors: volume change,
// momentum, then _apply_sources (k_li_cells' arithmetic).  own: its local index.
template <int KIND>
__device__ __forceinline__ void lt_cell(const LiArgs &q, const StepCtrl &s, const float4 st, const float4 ci, const float4 hz, float wt,
                                        float cl, const float4 *slots, const float *scale, int own, float &hn, float &hun, float &hvn,
                                        float (&led)[SURF_TERMS]) {
    const float dt = s.dt_f, md = q.md;
    const float own_scale = scale[own];
    float hd = 0.0f, qx = 0.0f, qy = 0.0f, bf = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 v = slots[k];
        const uint32_t b = __float_as_uint(v.w);
        if (!(b & LIS_PRESENT) || v.x == 0.0f) continue;
        if (b & LIS_INTERIOR) {
            const bool left = (b & LIS_LEFT) != 0;
            const float sd = (v.x >= 0.0f) != left ? scale[b >> 8] : own_scale;  // the donor's factor
            const float lim = v.x * sd * dt;
            hd += left ? -lim : lim;
        } else {
            const float bq = v.x * dt;
            hd -= bq;
            bf += bq;
        }
        qx += v.y;
        qy += v.z;
    }
    const float area = ci.x;
    const float h0 = fmax32(st.x + hd / area, 0.0f);
    const float per = 2.0f * area / fmax32(cl, 1.0e-12f);
    const bool wet0 = h0 > md;
    const float hu0 = wet0 ? qx / fmax32(per, 1.0e-12f) : 0.0f;
    const float hv0 = wet0 ? qy / fmax32(per, 1.0e-12f) : 0.0f;
    // _apply_sources (reference triangular_backend.py:1330-1379)
    const float rain = KIND == 1 ? s.rain_f * hz.w : s.rain_f;
    const float infil = KIND == 1 ? hz.y + (hz.x - hz.y) * __expf(-hz.z * wt) : q.infil_scalar;
    const float rd = fmax32(rain, 0.0f) * dt;
    const float h1 = h0 + rd;
    const float id = fmin32(h1, fmax32(infil, 0.0f) * dt);
    const float h2 = h1 - id;
    const float sc = (h1 > md) ? h2 / fmax32(h1, md) : 0.0f;
    const bool wet2 = h2 > md;
    hn = h2;
    hun = wet2 ? hu0 * sc : 0.0f;
    hvn = wet2 ? hv0 * sc : 0.0f;
    led[0] += rd * area;
    led[1] += id * area;
    led[3] += bf;
}

// Persistent and warp-specialised as k_surface: a producer warp fills two
// stages (bulk copies, then the halo states), eight compute warps run the
// tile's three passes; barriers full[2], halo[2], empty[2], pre (the first
// tile's static part, fetched before the wait for the previous kernel).  The
// last CTA plans the next step.
template <int KIND>
__global__ void __launch_bounds__(TILE + 32, 3) k_li_tiles(const __grid_constant__ LiTileArgs a, int slot, int plan_next) {
    extern __shared__ __align__(128) unsigned char smem[];
    float4 *s_slot = (float4 *)smem;                      // [(TILE + r1_cap) * 3]
    float *s_scale = (float *)(smem + a.off_scale);       // [TILE + r1_cap]
    int4 *s_info = (int4 *)(smem + a.off_bar + 64);       // [2][2]
    const uint32_t bar = smem_addr(smem + a.off_bar);
    const LiArgs &q = a.c;
    const int tid = threadIdx.x, ncta = (int)gridDim.x - 1;
    if ((int)blockIdx.x == ncta) {
        pdl_wait();
        if (a.early) pdl_launch_dependents();
        if (plan_next && tid == 0) plan_step(q.run, q.snap_t, q.hy, &q.ctrl[slot ^ 1], false, 0.0f, FL_PHASE_ALL);
        return;
    }
    const LtStage S0 = lt_stage(a, smem, 0), S1 = lt_stage(a, smem, 1);
    for (int i = tid; i < (TILE + a.r1_cap) * 3; i += TILE + 32) s_slot[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (tid == 0) {
        for (int k = 0; k < 2; ++k) {
            mbar_init(bar + 8u * k, 1);
            mbar_init(bar + 16u + 8u * k, 32);
            mbar_init(bar + 32u + 8u * k, TILE / 32);
        }
        mbar_init(bar + 48u, 1);
        mbar_fence_init();
    }
    __syncthreads();  // the last block-wide barrier: the roles split here
    if (tid == TILE) {  // (every CTA has a tile)
        const int4 ti = a.tile[2 * blockIdx.x], tj = a.tile[2 * blockIdx.x + 1];
        s_info[0] = ti;
        s_info[1] = tj;
        mbar_arrive_expect_tx(bar + 48u, lt_static_bytes<KIND>(ti, tj));
        lt_issue_static<KIND>(a, S0, ti, tj, bar + 48u, blockIdx.x);
    }
    pdl_wait();  // the previous step's kernels
    if (a.early) pdl_launch_dependents();
    const StepCtrl s = q.ctrl[slot];
    if (!s.active) {  // (uniform over the grid; no copy may land after the CTA leaves)
        if (tid == TILE && !mbar_wait_bounded(bar + 48u, 0, LT_WAIT_NS)) (void)mbar_wait_bounded(bar + 48u, 0, LT_WAIT_NS);
        return;
    }
    const float4 *__restrict__ in = s.parity ? q.state1 : q.state0;
    float4 *__restrict__ out = s.parity ? q.state0 : q.state1;

    if (tid >= TILE) {
        const int lane = tid - TILE;
        bool failed = false;
        int i = 0;
        for (int t = blockIdx.x; t < a.n_tiles; t += ncta, ++i) {
            const int st = i & 1;
            const LtStage &S = st ? S1 : S0;
            if (i >= 2) {
                bool ok = true;
                if (lane == 0) ok = mbar_wait_bounded(bar + 32u + 8u * st, ((i >> 1) - 1) & 1u, LT_WAIT_NS);
                if (!__shfl_sync(0xffffffffu, ok, 0)) {
                    failed = true;
                    break;
                }
            }
            if (lane == 0) {
                const uint32_t full = bar + 8u * st;
                if (i == 0) {
                    mbar_arrive_expect_tx(full, lt_step_bytes<KIND>());
                } else {
                    const int4 ti = a.tile[2 * t], tj = a.tile[2 * t + 1];
                    s_info[2 * st] = ti;
                    s_info[2 * st + 1] = tj;
                    mbar_arrive_expect_tx(full, lt_static_bytes<KIND>(ti, tj) + lt_step_bytes<KIND>());
                    lt_issue_static<KIND>(a, S, ti, tj, full, t);
                }
                lt_issue_step<KIND>(in, q.wet, S, full, t);
            }
            const uint32_t lbar = i == 0 ? bar + 48u : bar + 8u * st;
            const uint32_t lpar = i == 0 ? 0u : (uint32_t)((i >> 1) & 1);
            const bool ok = mbar_wait_bounded(lbar, lpar, LT_WAIT_NS);
            if (!__all_sync(0xffffffffu, ok)) {
                // a copy is late: one more bounded wait so none lands after the CTA leaves
                (void)mbar_wait_bounded(lbar, lpar, LT_WAIT_NS);
                if (i == 0) (void)mbar_wait_bounded(bar + 8u * st, 0u, LT_WAIT_NS);
                failed = true;
                break;
            }
            const int hc = s_info[2 * st].w;
            for (int j = lane; j < hc; j += 32) cp_async16(smem_addr(&S.st[TILE + j]), in + S.hs[j]);
            cp_async_arrive_noinc(bar + 16u + 8u * st);
        }
        cp_async_wait_all();
        if (failed && lane == 0) {
            if (atomicCAS(&q.run->error, 0, FL_E_TIMEOUT) == 0) q.run->error_step = s.step;
        }
        return;
    }

    const float dt = s.dt_f, md = q.md;
    const bool do_surface = (s.phases & FL_PHASE_SURFACE) != 0;
    const bool drain_finishes = (s.phases & FL_PHASE_DRAINAGE) != 0;
    const bool recharge_finishes = (s.phases & FL_PHASE_RECHARGE) != 0;
    float led[SURF_TERMS] = {0.0f, 0.0f, 0.0f, 0.0f};
    const int led_warp = (int)blockIdx.x * (TILE / 32) + (tid >> 5);
    const float2 slots = ledger_fetch<SURF_TERMS>(q.ledger, led_warp);
    int i = 0;
    for (int t = blockIdx.x; t < a.n_tiles; t += ncta, ++i) {
        const int st_i = i & 1;
        const LtStage &S = st_i ? S1 : S0;
        bool ok = true;
        if (tid == 0)
            ok = (i > 0 || mbar_wait_bounded(bar + 48u, 0u, LT_WAIT_NS)) &&
                 mbar_wait_bounded(bar + 8u * st_i, (i >> 1) & 1u, LT_WAIT_NS) &&
                 mbar_wait_bounded(bar + 16u + 8u * st_i, (i >> 1) & 1u, LT_WAIT_NS);
        if (!lt_all(ok)) {
            if (tid == 0 && atomicCAS(&q.run->error, 0, FL_E_TIMEOUT) == 0) q.run->error_step = s.step;
            break;  // the producer waits out its own copies
        }
        const int n1 = s_info[2 * st_i + 1].x;
        const float4 ci = S.ci[tid];
        if (do_surface) {
            const int n_e = s_info[2 * st_i].y;
#pragma unroll 1
            for (int e = tid; e < n_e; e += TILE) lt_entry(S.en[e], S.dm[e], S.st, s_slot, q.g, dt);
            lt_sync();  // the discharges are in place
            s_scale[tid] = lt_donor_scale(&s_slot[tid * 3], S.st[tid].x, ci.x, dt);
            for (int k = tid; k < n1; k += TILE)
                s_scale[TILE + k] = lt_donor_scale(&s_slot[(TILE + k) * 3], S.st[TILE + k].x, S.ha[k], dt);
            lt_sync();  // the donor factors are in place
        }
        const int c = t * TILE + tid;
        if (c < q.C) {
            const float4 st = S.st[tid];
            const uint32_t info = __float_as_uint(ci.z);
            if (s.check_finite && !isfinite(st.x)) {
                if (atomicCAS(&q.run->error, 0, FL_E_NONFINITE) == 0) q.run->error_step = s.step;
            }
            float wt = 0.0f;
            float4 hz = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
            if (KIND == 1) {
                wt = S.wt[tid];
                hz = S.hz[tid];
            }
            float hn = 0.0f, hun = 0.0f, hvn = 0.0f;
            if (!do_surface) {
                hn = st.x; hun = st.y; hvn = st.z;
            } else if (info & CELL_ACTIVE) {
                lt_cell<KIND>(q, s, st, ci, hz, wt, S.cl[tid], &s_slot[tid * 3], s_scale, tid, hn, hun, hvn, led);
            }
            if (s.phases & FL_PHASE_CLAMP) clamp_velocity_exact(hn, hun, hvn, q.vmax);
            if ((info & CELL_RECEIVER) && (s.phases & FL_PHASE_INFLOW)) hn = __fadd_rn(hn, q.ext_add[c]);
            out[c] = make_float4(hn, hun, hvn, st.w);
            const bool final_here = !(drain_finishes && (info & CELL_COUPLED)) &&
                                    !(recharge_finishes && (info & CELL_RECHARGE));
            if (KIND == 1 && do_surface && final_here) q.wet[c] = wt + dt * (float)(hn > md);
            if (s.snap_slot >= 0) {
                const size_t o = (size_t)s.snap_slot * (size_t)q.C + (size_t)c;
                if (final_here) q.snap_h[o] = hn;
                q.snap_hu[o] = hun;
                q.snap_hv[o] = hvn;
            }
        }
        // the places are empty again for the next tile (its entries are written
        // after its opening barrier)
#pragma unroll
        for (int k = 0; k < 3; ++k) s_slot[tid * 3 + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int k = tid; k < n1 * 3; k += TILE) s_slot[TILE * 3 + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(bar + 32u + 8u * st_i);
    }
    ledger_add<SURF_TERMS>(led, slots, q.ledger, led_warp);
}

// `steps` steps of a run of the local-inertial surface alone in one cooperative
// launch (fl_run.cuh), a CTA a tile: k_li_tiles' three passes on a tile that stays in
// shared memory and registers, with its ledger slots and order.  us a step of a whole
// run with 32 steps between CFL evaluations, a launch a step -> here: 1,800 cells 4.7
// -> 3.4, 20,000 cells 5.0 -> 3.8, 105,800 cells 6.6 -> 4.8; what is left is the halo
// states' round trip and the three passes.
template <int KIND>
__global__ void __launch_bounds__(RUN_THREADS, 3) k_li_run(const __grid_constant__ LiTileArgs a, const RunArgs x, int slot, int steps) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ StepCtrl s_ctrl[2];
    __shared__ RunCtrl s_run;
    float4 *s_slot = (float4 *)smem;
    float *s_scale = (float *)(smem + a.off_scale);
    const uint32_t bar = smem_addr(smem + a.off_bar);
    const LiArgs &q = a.c;
    const int tid = threadIdx.x, tile = blockIdx.x, n_tiles = a.n_tiles;
    uint32_t *mine = x.serial + (size_t)tile * SYNC_STRIDE;
    const uint32_t base = *mine;
    const StepCtrl first = q.ctrl[slot];
    if (!first.active) {  // (uniform over the grid)
        if (tid == 0) publish(mine, base + steps);
        return;
    }
    if (tile == n_tiles) {
        run_last_cta(q.run, q.ctrl, q.snap_t, q.hy, x, n_tiles, base, steps, first, &s_run, &s_ctrl[1]);
        return;
    }
    const LtStage S = lt_stage(a, smem, 0);
    const int4 ti = a.tile[2 * tile], tj = a.tile[2 * tile + 1];
    const int n1 = tj.x;
    for (int i = tid; i < (TILE + n1) * 3; i += RUN_THREADS) s_slot[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
        mbar_arrive_expect_tx(bar, lt_static_bytes<KIND>(ti, tj) + lt_step_bytes<KIND>());
        lt_issue_static<KIND>(a, S, ti, tj, bar, tile);
        lt_issue_step<KIND>(first.parity ? q.state1 : q.state0, q.wet, S, bar, tile);
        s_ctrl[0] = first;
        s_run = *q.run;
        s_run.error = 0;  // (a tile that is ahead may have set it)
    }
    __syncthreads();
    // every thread has read its serial number and the first record, this one the run control
    if (tid == 0) publish(mine, base + steps);
    bool ok = mbar_wait_bounded(bar, 0, LT_WAIT_NS);
    if (!ok) ok = mbar_wait_bounded(bar, 0, LT_WAIT_NS);  // none may land after the CTA leaves
    if (tid >= TILE) {
        run_records(ok, steps, q.hy, q.run, n_tiles, &s_run, s_ctrl);
        return;
    }

    float2 total[SURF_TERMS];  // lane 0 of a warp: its ledger sums
    float2 *ledger = q.ledger + (size_t)(tile * (TILE / 32) + (tid >> 5)) * SURF_TERMS;
#pragma unroll
    for (int j = 0; j < SURF_TERMS; ++j) total[j] = (tid & 31) == 0 ? ledger[j] : make_float2(0.0f, 0.0f);
    const int c = tile * TILE + tid;
    const float4 ci = S.ci[tid];
    const uint32_t info = __float_as_uint(ci.z);
    const bool sent = (x.sent[c >> 5] >> (c & 31) & 1u) != 0;  // another tile reads the cell
    const float cl = S.cl[tid];
    float wt = 0.0f;
    float4 hz = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
    if (KIND == 1) {
        wt = S.wt[tid];
        hz = S.hz[tid];
    }
    int k = 0;
    for (; k < steps; ++k) {
        ok = run_halo(ok, k, first.parity ? q.state1 : q.state0, x, base, S.hs, ti.w, S.st);
        if (!run_all(ok)) {  // the halo states and the step record are in place
            if (tid == 0 && atomicCAS(&q.run->error, 0, FL_E_TIMEOUT) == 0) q.run->error_step = first.step + k;
            break;
        }
        const StepCtrl s = s_ctrl[k & 1];
        if (!s.active) break;  // (uniform over the grid)
        const float dt = s.dt_f;
        const bool do_surface = (s.phases & FL_PHASE_SURFACE) != 0;
        float led[SURF_TERMS] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (do_surface) {
#pragma unroll 1
            for (int e = tid; e < ti.y; e += TILE) lt_entry(S.en[e], S.dm[e], S.st, s_slot, q.g, dt);
            lt_sync();  // the discharges are in place
            s_scale[tid] = lt_donor_scale(&s_slot[tid * 3], S.st[tid].x, ci.x, dt);
            for (int j = tid; j < n1; j += TILE)
                s_scale[TILE + j] = lt_donor_scale(&s_slot[(TILE + j) * 3], S.st[TILE + j].x, S.ha[j], dt);
        }
        lt_sync();  // the donor factors are in place
        if (c < q.C) {
            const float4 st = S.st[tid];
            if (s.check_finite && !isfinite(st.x)) run_non_finite(q.run, s.step);
            float hn = 0.0f, hun = 0.0f, hvn = 0.0f;
            if (!do_surface) {
                hn = st.x; hun = st.y; hvn = st.z;
            } else if (info & CELL_ACTIVE) {
                lt_cell<KIND>(q, s, st, ci, hz, wt, cl, &s_slot[tid * 3], s_scale, tid, hn, hun, hvn, led);
            }
            if (s.phases & FL_PHASE_CLAMP) clamp_velocity_exact(hn, hun, hvn, q.vmax);
            if (sent) send_state(x.exchange + (size_t)((base + k + 1) & 1u) * x.cells + c, hn, hun, hvn, base + k + 1);
            S.st[tid] = make_float4(hn, hun, hvn, st.w);
            if (KIND == 1 && do_surface) wt = wt + dt * (float)(hn > q.md);
            if (s.snap_slot >= 0) {
                const size_t o = (size_t)s.snap_slot * (size_t)q.C + (size_t)c;
                q.snap_h[o] = hn;
                q.snap_hu[o] = hun;
                q.snap_hv[o] = hvn;
            }
        }
        // the places are empty again for the next step (its entries are written after
        // the barrier that follows its halo)
#pragma unroll
        for (int j = 0; j < 3; ++j) s_slot[tid * 3 + j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int j = tid; j < n1 * 3; j += TILE) s_slot[TILE * 3 + j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < SURF_TERMS; ++j) {
            float y = led[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) y += __shfl_down_sync(0xffffffffu, y, o);
            if ((tid & 31) == 0) ff_accumulate(&total[j], y);
        }
    }
    // k steps were run: the states go where the next launch reads them
    if (c < q.C) {
        if (k > 0) (((first.parity ^ k) & 1) ? q.state1 : q.state0)[c] = S.st[tid];
        if (KIND == 1) q.wet[c] = wt;
    }
    if ((tid & 31) == 0) {
#pragma unroll
        for (int j = 0; j < SURF_TERMS; ++j) ledger[j] = total[j];
    }
}

// Shared memory layout and grid of k_li_tiles; 0 blocks where fewer than two
// CTAs fit an SM (the two launches are then the better choice).
cudaError_t plan_li_tiles(LiTileArgs &a, int kind, int device, int *grid, int *smem_bytes) {
    auto up = [](int x, int m) { return (x + m - 1) / m * m; };
    a.off_scale = (TILE + a.r1_cap) * 48;
    a.off_bar = up(a.off_scale + (TILE + a.r1_cap) * 4, 128);
    a.off_stage = a.off_bar + 128;  // seven barriers, two tile records of 32 bytes at 64
    int o = (TILE + a.h_cap) * 16;
    a.so_ci = o;
    o += TILE * 16;
    a.so_hz = o;
    if (kind) o += TILE * 16;
    a.so_en = o;
    o += a.e_cap * 16;
    a.so_dm = o;
    o += a.e_cap * 8;
    a.so_wt = o;
    if (kind) o += TILE * 4;
    a.so_cl = o;
    o += TILE * 4;
    a.so_hs = o;
    o += up(a.h_cap, 4) * 4;
    a.so_ha = o;
    o += up(a.r1_cap, 4) * 4;
    a.stage_bytes = up(o, 128);
    *smem_bytes = a.off_stage + 2 * a.stage_bytes;
    *grid = 0;
    const void *fn = kind ? (const void *)k_li_tiles<1> : (const void *)k_li_tiles<0>;
    int per_sm = 0, sms = 0, most = 0;
    cudaError_t e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return e;
    if (*smem_bytes > most) return cudaSuccess;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, TILE + 32, (size_t)*smem_bytes);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess || per_sm < 2) return e;
    *grid = std::max(1, std::min(per_sm * sms - 1, a.n_tiles)) + 1;
    a.early = 2 * *grid <= per_sm * sms ? 1 : 0;
    return cudaSuccess;
}

cudaError_t launch_li_tiles(const LiTileArgs &a, int kind, int slot, int plan_next, int grid, int smem_bytes,
                            cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(TILE + 32);
    cfg.dynamicSmemBytes = (size_t)smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return kind == 1 ? cudaLaunchKernelEx(&cfg, k_li_tiles<1>, a, slot, plan_next)
                     : cudaLaunchKernelEx(&cfg, k_li_tiles<0>, a, slot, plan_next);
}

// Whether k_li_run can run the mesh: a CTA per tile of k_li_tiles' grid and all
// resident at once.  *smem_bytes 0: it cannot.
cudaError_t plan_li_run(const LiTileArgs &a, int kind, int tiles_grid, int device, int *smem_bytes, size_t *serial_words) {
    const void *fn = kind ? (const void *)k_li_run<1> : (const void *)k_li_run<0>;
    const int bytes = a.off_stage + a.stage_bytes;
    *smem_bytes = 0;
    *serial_words = (size_t)(a.n_tiles + 1) * SYNC_STRIDE;
    if (a.n_tiles + 1 != tiles_grid) return cudaSuccess;
    return run_fits(fn, a.n_tiles + 1, bytes, device, smem_bytes);
}

cudaError_t launch_li_run(const LiTileArgs &a, int kind, const RunArgs &x, int slot, int steps, int smem_bytes, cudaStream_t stream) {
    return launch_run(kind ? k_li_run<1> : k_li_run<0>, a, x, slot, steps, a.n_tiles + 1, smem_bytes, stream);
}

int li_edge_blocks(int32_t E, int sms) { return std::max(1, std::min(sms * 8, (E + 255) / 256)); }
int li_cell_blocks(int32_t C) { return (C + 255) / 256 + 1; }  // + the planner block

// Both launched as programmatic dependents of the kernel before them, so
// each one's launch overlaps the end of the previous one.
cudaError_t launch_li(const LiArgs &a, int kind, int slot, int plan_next, int sms, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3((unsigned)li_edge_blocks(a.E, sms));
    cudaError_t e = cudaLaunchKernelEx(&cfg, k_li_edges, a, slot);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3((unsigned)li_cell_blocks(a.C));
    return kind == 1 ? cudaLaunchKernelEx(&cfg, k_li_cells<1>, a, slot, plan_next)
                     : cudaLaunchKernelEx(&cfg, k_li_cells<0>, a, slot, plan_next);
}

}  // namespace fl
