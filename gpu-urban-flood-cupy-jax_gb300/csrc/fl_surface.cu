// Surface kernels for sm_103a.
//
// k_surface: a persistent, warp-specialised kernel.  Each CTA walks its tiles
// (256 consecutive Hilbert-ordered cells each) through a two-stage
// shared-memory pipeline: a producer warp has the bulk-copy (TMA) engine
// bring a tile's contiguous blocks -- states, cell info, Horton fields, wet
// time, the edge entries and the halo cell list -- into a stage and then
// gathers its halo states with cp.async, while eight compute warps work on
// the other stage, so DRAM latency overlaps the arithmetic.  Per tile:
//   phase 2  every edge entry of the tile once -- ghost state, hydrostatic
//            reconstruction, HLL (reference triangular_swe_cuda_kernels.py
//            :22-203, equations.py:20-152, triangular_backend.py:1067-1178,
//            1294-1327) -- each cell's share written to its (cell, slot)
//            place in shared memory (one writer per place: no atomics);
//   phase 3  each thread sums its cell's slots in the reference's order and
//            does the cell update with Manning damping (:206-252), rainfall
//            and infiltration (triangular_backend.py:1330-1379), the velocity
//            clamp (solver/stabilizers.py:8-27), external inflow, wet time,
//            snapshot writes and the ledger.  (The inlet requests of inlet
//            cells are evaluated by k_nodes from this kernel's output.)
// An edge between two tiles is evaluated in each (same code, same inputs),
// so its two cells always apply the same mass flux: the scheme is exactly
// conservative and bitwise reproducible.  The last CTA of the grid only plans
// the next step (a single thread of float64 control arithmetic that would
// otherwise delay one CTA's tiles).
//
// The flux arithmetic uses reciprocal-based division and fast exp/log (it is
// instruction-bound); values stay within a few ulp of the reference's
// correctly rounded float32 operations.  The velocity clamp and the CFL dt use
// correctly rounded, uncontracted operations and match the reference
// bit-for-bit.
//
// k_dt: the global CFL minimum (equations.py:155-178) as a warp-shuffle and
// single-pass grid reduction; the last block to finish plans the step.
#include <algorithm>

#include "fl_device.cuh"
#include "fl_run.cuh"

namespace fl {

int surface_smem_layout(SurfArgs &a, int kind);

constexpr uint64_t COPY_WAIT_NS = 1000000000ull;  // 1 s per wait on a tile copy

struct TileStage {
    float4 *st;         // [TILE + h_cap] own states then halo states
    float4 *ci;         // [TILE]
    float4 *hz;         // [TILE] (kind 1)
    float *wt;          // [TILE] (kind 1)
    float4 *en;         // [e_cap]
    int32_t *hs;        // [h_cap]
};

__device__ __forceinline__ TileStage stage_at(const SurfArgs &a, unsigned char *smem, int s) {
    unsigned char *b = smem + a.off_stage + s * a.stage_bytes;
    TileStage t;
    t.st = (float4 *)b;
    t.ci = (float4 *)(b + a.so_ci);
    t.hz = (float4 *)(b + a.so_hz);
    t.wt = (float *)(b + a.so_wt);
    t.en = (float4 *)(b + a.so_en);
    t.hs = (int32_t *)(b + a.so_hs);
    return t;
}

// Issue the bulk copies of tile t into a stage (one thread): the static part
// (cell info, Horton fields, entries, halo list) and the part that a step
// writes (states, wet time).  The byte count a barrier expects is the sum of
// exactly the copies issued for it.
template <int KIND>
__device__ __forceinline__ uint32_t static_bytes(const int4 ti) {
    return TILE * 16u + (KIND == 1 ? TILE * 16u : 0u) + (uint32_t)ti.y * 16u + (uint32_t)((ti.w + 3) & ~3) * 4u;
}
template <int KIND>
__device__ __forceinline__ uint32_t step_bytes() {
    return TILE * 16u + (KIND == 1 ? TILE * 4u : 0u);
}

template <int KIND>
__device__ __forceinline__ void issue_static(const SurfArgs &a, const TileStage &S, const int4 ti, uint32_t bar, int t) {
    const uint32_t ent_bytes = (uint32_t)ti.y * 16u;
    const uint32_t halo_bytes = (uint32_t)((ti.w + 3) & ~3) * 4u;
    const size_t c0 = (size_t)t * TILE;
    bulk_copy_g2s(smem_addr(S.ci), a.cinfo + c0, TILE * 16u, bar);
    if (KIND == 1) bulk_copy_g2s(smem_addr(S.hz), a.horton + c0, TILE * 16u, bar);
    if (ent_bytes) bulk_copy_g2s(smem_addr(S.en), a.ent + ti.x, ent_bytes, bar);
    if (halo_bytes) bulk_copy_g2s(smem_addr(S.hs), a.halo_src + ti.z, halo_bytes, bar);
}

template <int KIND>
__device__ __forceinline__ void issue_step(const float4 *in, const float *wet, const TileStage &S, uint32_t bar, int t) {
    const size_t c0 = (size_t)t * TILE;
    bulk_copy_g2s(smem_addr(S.st), in + c0, TILE * 16u, bar);
    if (KIND == 1) bulk_copy_g2s(smem_addr(S.wt), wet + c0, TILE * 4u, bar);
}

// Named barrier and barrier-reduction among the compute warps only (id 1).
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(TILE) : "memory"); }

__device__ __forceinline__ bool compute_all(bool p) {
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

// Warp-specialised persistent surface kernel: 8 compute warps (one thread
// per cell of a 256-cell tile) and one producer warp.  The producer fills the
// two stages: bulk copies (TMA engine) of a tile's states, cell info, Horton
// fields, wet time, edge entries and halo list onto stage barrier full[s],
// then, once they land, the halo state gathers (cp.async, one arrive per lane
// on halo[s] when they land).  The compute warps wait on full[s] and halo[s],
// run phase 2 (each edge entry once: flux into per-(cell, slot) places) and
// phase 3 (the cell update), and release the stage on empty[s].  Loads of
// the next tile therefore overlap both compute phases of the current one.
// Every wait is bounded (1 s): a timeout records FL_E_TIMEOUT and the CTA
// leaves after its copies in flight have landed (or a second bounded wait).
//
// The static part of a CTA's first tile is fetched before the wait for the
// step's previous kernel (barrier pre).  A grid that leaves CTA slots free
// (a.early) also lets its dependent start once its own wait is over: the next
// kernel's CTAs are then set up, with that fetch done, when this one ends.
// (A grid that fills the device does not: CTAs waiting next to it cost more
// than the launch latency they hide.)  Ensemble members (MEM): one launch,
// blockIdx.y = member, each with the grid of a single run.
template <int KIND, bool MEM>
__global__ void __launch_bounds__(SURF_THREADS, 4) k_surface(const __grid_constant__ SurfArgs a, int slot, int plan_next) {
    extern __shared__ __align__(128) unsigned char smem[];
    float4 *s_flux = (float4 *)smem;  // [TILE * 3] per (cell, slot): {mass, x-mom, y-mom} x len
    uint64_t *s_bar = (uint64_t *)(smem + a.off_bar);  // full[2], halo[2], empty[2], pre
    int4 *s_info = (int4 *)(smem + a.off_bar + 64);
    const int tid = threadIdx.x;
    const int ncta = (int)gridDim.x - 1;  // the last CTA plans
    const size_t mem = MEM ? blockIdx.y : 0;
    RunCtrl *run = a.run + mem;
    const StepCtrl *ctrl = a.ctrl + 2 * mem;
    if ((int)blockIdx.x == ncta) {
        pdl_wait();
        if (a.early) pdl_launch_dependents();
        if (plan_next && tid == 0)
            plan_step(run, a.snap_t + mem * (size_t)a.max_snaps, MEM ? a.hys[mem] : a.hy, &a.ctrl[2 * mem + (slot ^ 1)],
                      false, 0.0f, FL_PHASE_ALL);
        return;
    }
    // barrier addresses: full(s) = base + 8 s, halo(s) = base + 16 + 8 s, empty(s) = base + 32 + 8 s, pre = base + 48
    const uint32_t bar_base = smem_addr(s_bar);
    const TileStage S0 = stage_at(a, smem, 0), S1 = stage_at(a, smem, 1);
    if (tid < TILE) {
#pragma unroll
        for (int k = 0; k < 3; ++k) s_flux[tid * 3 + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (tid == 0) {
        for (int k = 0; k < 2; ++k) {
            mbar_init(bar_base + 8u * k, 1);
            mbar_init(bar_base + 16u + 8u * k, 32);
            mbar_init(bar_base + 32u + 8u * k, TILE / 32);  // one arrival per compute warp
        }
        mbar_init(bar_base + 48u, 1);
        mbar_fence_init();
    }
    __syncthreads();  // the last block-wide barrier: the roles split here
    if (tid == TILE) {  // (every CTA has a tile)
        const int4 ti = a.tile_info[blockIdx.x];
        s_info[0] = ti;
        mbar_arrive_expect_tx(bar_base + 48u, static_bytes<KIND>(ti));
        issue_static<KIND>(a, S0, ti, bar_base + 48u, blockIdx.x);
    }
    // launched as a programmatic dependent of the step's previous kernel: the
    // set-up above overlaps its end; the step record, the states and the wet
    // time it (or an earlier kernel) wrote are read after this wait
    pdl_wait();
    if (a.early) pdl_launch_dependents();
    const StepCtrl s = ctrl[slot];
    if (!s.active) {  // (uniform over the member's grid; no copy may land after the CTA leaves)
        if (tid == TILE && !mbar_wait_bounded(bar_base + 48u, 0, COPY_WAIT_NS))
            (void)mbar_wait_bounded(bar_base + 48u, 0, COPY_WAIT_NS);
        return;
    }
    const size_t mc = MEM ? mem * (size_t)a.m_cells : 0;
    const float4 *__restrict__ in = (s.parity ? a.state1 : a.state0) + mc;
    float4 *__restrict__ out = (s.parity ? a.state0 : a.state1) + mc;
    float *__restrict__ wet = a.wet + mc;

    if (tid >= TILE) {
        // ---------------------------------------------------------- producer
        const int lane = tid - TILE;
        bool failed = false;
        int i = 0;
        for (int t = blockIdx.x; t < a.n_tiles; t += ncta, ++i) {
            const int st = i & 1;
            const TileStage &S = st ? S1 : S0;
            if (i >= 2) {  // the compute warps released this stage's previous tile
                bool ok = true;
                if (lane == 0) ok = mbar_wait_bounded((bar_base + 32u + 8u * st), ((i >> 1) - 1) & 1u, COPY_WAIT_NS);
                if (!__shfl_sync(0xffffffffu, ok, 0)) {
                    failed = true;
                    break;
                }
            }
            if (lane == 0) {
                const uint32_t bar = bar_base + 8u * st;
                if (i == 0) {
                    mbar_arrive_expect_tx(bar, step_bytes<KIND>());
                } else {
                    const int4 ti = a.tile_info[t];
                    s_info[st] = ti;
                    mbar_arrive_expect_tx(bar, static_bytes<KIND>(ti) + step_bytes<KIND>());
                    issue_static<KIND>(a, S, ti, bar, t);
                }
                issue_step<KIND>(in, wet, S, bar, t);
            }
            // every lane waits: each then reads the landed halo list itself
            // (the first tile's landed on pre; its gathers go out before its states are in)
            const uint32_t lbar = i == 0 ? bar_base + 48u : bar_base + 8u * st;
            const uint32_t lpar = i == 0 ? 0u : (uint32_t)((i >> 1) & 1);
            const bool ok = mbar_wait_bounded(lbar, lpar, COPY_WAIT_NS);
            if (!__all_sync(0xffffffffu, ok)) {
                // a copy is late: one more bounded wait so none lands after the CTA leaves
                (void)mbar_wait_bounded(lbar, lpar, COPY_WAIT_NS);
                if (i == 0) (void)mbar_wait_bounded(bar_base + 8u * st, 0u, COPY_WAIT_NS);
                failed = true;
                break;
            }
            const int hc = s_info[st].w;
            for (int j = lane; j < hc; j += 32) cp_async16(smem_addr(&S.st[TILE + j]), in + S.hs[j]);
            cp_async_arrive_noinc((bar_base + 16u + 8u * st));
        }
        cp_async_wait_all();
        if (failed && lane == 0) {
            if (atomicCAS(&run->error, 0, FL_E_TIMEOUT) == 0) run->error_step = s.step;
        }
        return;
    }

    // ------------------------------------------------------------- compute
    const float dt = s.dt_f;
    const float md = a.md;
    const bool do_surface = (s.phases & FL_PHASE_SURFACE) != 0;
    const bool drain_finishes = (s.phases & FL_PHASE_DRAINAGE) != 0;
    const bool recharge_finishes = (s.phases & FL_PHASE_RECHARGE) != 0;
    float led[SURF_TERMS] = {0.0f, 0.0f, 0.0f, 0.0f};
    float2 *ledger = a.ledger + (MEM ? mem * (size_t)a.m_led : 0);
    const int led_warp = (int)blockIdx.x * (TILE / 32) + (tid >> 5);
    const float2 slots = ledger_fetch<SURF_TERMS>(ledger, led_warp);
    int i = 0;
    for (int t = blockIdx.x; t < a.n_tiles; t += ncta, ++i) {
        const int st_i = i & 1;
        const TileStage &S = st_i ? S1 : S0;
        // one thread waits for the tile's copies and gathers; the barrier
        // reduction hands them to the other compute threads
        bool ok = true;
        if (tid == 0)
            ok = (i > 0 || mbar_wait_bounded(bar_base + 48u, 0u, COPY_WAIT_NS)) &&
                 mbar_wait_bounded((bar_base + 8u * st_i), (i >> 1) & 1u, COPY_WAIT_NS) &&
                 mbar_wait_bounded((bar_base + 16u + 8u * st_i), (i >> 1) & 1u, COPY_WAIT_NS);
        if (!compute_all(ok)) {
            if (tid == 0 && atomicCAS(&run->error, 0, FL_E_TIMEOUT) == 0) run->error_step = s.step;
            break;  // the producer waits out its own copies
        }

        // phase 2: each edge entry of the tile once
        const int c0 = t * TILE;
        if (do_surface) {
            const int n_e = s_info[st_i].y;
#pragma unroll 1
            for (int e = tid; e < n_e; e += TILE)
                tile_entry(S.en[e], S.st, s_flux, a.g, a.half_g, md, a.stage, dt, led[2], led[3]);
        }
        compute_sync();  // phase 2's slots are complete

        // phase 3: the cell update
        const int c = c0 + tid;
        if (c < a.C) {
            const float4 st = S.st[tid];
            const float4 ci = S.ci[tid];
            const uint32_t info = __float_as_uint(ci.z);
            if (s.check_finite && !isfinite(st.x)) {
                if (atomicCAS(&run->error, 0, FL_E_NONFINITE) == 0) run->error_step = s.step;
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
                const float rain = KIND == 1 ? s.rain_f * hz.w : s.rain_f;
                const float infil = KIND == 1 ? hz.y + (hz.x - hz.y) * __expf(-hz.z * wt) : a.infil_scalar;
                const CellNew u = cell_update(st, ci, &s_flux[tid * 3], dt, s.dtg_f, md, rain, infil);
                hn = u.h; hun = u.hu; hvn = u.hv;
                led[0] += u.rd * ci.x;
                led[1] += u.id * ci.x;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) s_flux[tid * 3 + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (s.phases & FL_PHASE_CLAMP) clamp_velocity_exact(hn, hun, hvn, a.vmax);
            // external boundary inflow after the clamp (reference engine.py:263-273)
            if ((info & CELL_RECEIVER) && (s.phases & FL_PHASE_INFLOW)) hn = __fadd_rn(hn, a.ext_add[c]);
            out[c] = make_float4(hn, hun, hvn, st.w);
            const bool final_here = !(drain_finishes && (info & CELL_COUPLED)) &&
                                    !(recharge_finishes && (info & CELL_RECHARGE));
            if (KIND == 1 && do_surface && final_here) wet[c] = wt + dt * (float)(hn > md);
            if (s.snap_slot >= 0) {
                const size_t o = (MEM ? mem * (size_t)a.m_snap : 0) + (size_t)s.snap_slot * (size_t)a.C + (size_t)c;
                if (final_here) a.snap_h[o] = hn;
                a.snap_hu[o] = hun;
                a.snap_hv[o] = hvn;
            }
        }
        // each compute warp releases the stage once its lanes are done with it;
        // the flux slots need no barrier here: the next tile's phase 2 writes
        // them only after its opening barrier reduction, which every compute
        // thread reaches after this phase 3
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive((bar_base + 32u + 8u * st_i));
    }
    ledger_add<SURF_TERMS>(led, slots, ledger, led_warp);
}

// `steps` steps of a run of the surface alone in one cooperative launch (fl_run.cuh):
// a tile's entries, halo list, cell data, wet time and states stay in shared memory
// and registers.  The ledger sums keep k_surface's slots and order: the same bits,
// step by step.
//
// A launch a step costs a small mesh more than its work.  us a step of a whole run
// with 32 (8) steps between CFL evaluations, a launch a step -> here: 1,800 cells
// 3.8 -> 3.0 (4.5 -> 4.0), 20,000 cells 3.8 -> 3.0 (4.5 -> 3.8), 153,458 cells 5.6 ->
// 4.5 (6.6 -> 5.7); what is left is the halo states' round trip and the two phases.
template <int KIND>
__global__ void __launch_bounds__(RUN_THREADS, 4) k_surface_run(const __grid_constant__ SurfArgs a, const RunArgs x, int slot, int steps) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ StepCtrl s_ctrl[2];
    __shared__ RunCtrl s_run;
    float4 *s_flux = (float4 *)smem;
    const uint32_t bar = smem_addr(smem + a.off_bar);
    const int tid = threadIdx.x, tile = blockIdx.x, n_tiles = a.n_tiles;
    uint32_t *mine = x.serial + (size_t)tile * SYNC_STRIDE;
    const uint32_t base = *mine;
    const StepCtrl first = a.ctrl[slot];
    if (!first.active) {  // (uniform over the grid)
        if (tid == 0) publish(mine, base + steps);
        return;
    }
    if (tile == n_tiles) {
        run_last_cta(a.run, a.ctrl, a.snap_t, a.hy, x, n_tiles, base, steps, first, &s_run, &s_ctrl[1]);
        return;
    }
    const TileStage S = stage_at(a, smem, 0);
    const int4 ti = a.tile_info[tile];
    for (int i = tid; i < TILE * 3; i += RUN_THREADS) s_flux[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
        mbar_arrive_expect_tx(bar, static_bytes<KIND>(ti) + step_bytes<KIND>());
        issue_static<KIND>(a, S, ti, bar, tile);
        issue_step<KIND>(first.parity ? a.state1 : a.state0, a.wet, S, bar, tile);
        s_ctrl[0] = first;
        s_run = *a.run;
        s_run.error = 0;  // (a tile that is ahead may have set it)
    }
    __syncthreads();
    // every thread has read its serial number and the first record, this one the run control
    if (tid == 0) publish(mine, base + steps);
    bool ok = mbar_wait_bounded(bar, 0, COPY_WAIT_NS);
    if (!ok) ok = mbar_wait_bounded(bar, 0, COPY_WAIT_NS);  // none may land after the CTA leaves

    if (tid >= TILE) {
        run_records(ok, steps, a.hy, a.run, n_tiles, &s_run, s_ctrl);
        return;
    }

    float2 total[SURF_TERMS];  // lane 0 of a warp: its ledger sums
    float2 *ledger = a.ledger + (size_t)(tile * (TILE / 32) + (tid >> 5)) * SURF_TERMS;
#pragma unroll
    for (int j = 0; j < SURF_TERMS; ++j) total[j] = (tid & 31) == 0 ? ledger[j] : make_float2(0.0f, 0.0f);
    const int c = tile * TILE + tid;
    const float4 ci = S.ci[tid];
    const uint32_t info = __float_as_uint(ci.z);
    const bool sent = (x.sent[c >> 5] >> (c & 31) & 1u) != 0;  // another tile reads the cell
    float wt = 0.0f;
    float4 hz = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
    if (KIND == 1) {
        wt = S.wt[tid];
        hz = S.hz[tid];
    }
    const float md = a.md;
    int k = 0;
    for (; k < steps; ++k) {
        ok = run_halo(ok, k, first.parity ? a.state1 : a.state0, x, base, S.hs, ti.w, S.st);
        if (!run_all(ok)) {  // the halo states and the step record are in place
            if (tid == 0 && atomicCAS(&a.run->error, 0, FL_E_TIMEOUT) == 0) a.run->error_step = first.step + k;
            break;
        }
        const StepCtrl s = s_ctrl[k & 1];
        if (!s.active) break;  // (uniform over the grid)
        const float dt = s.dt_f;
        const bool do_surface = (s.phases & FL_PHASE_SURFACE) != 0;
        float led[SURF_TERMS] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (do_surface) {
#pragma unroll 1
            for (int e = tid; e < ti.y; e += TILE)
                tile_entry(S.en[e], S.st, s_flux, a.g, a.half_g, md, a.stage, dt, led[2], led[3]);
        }
        compute_sync();
        if (c < a.C) {
            const float4 st = S.st[tid];
            if (s.check_finite && !isfinite(st.x)) run_non_finite(a.run, s.step);
            float hn = 0.0f, hun = 0.0f, hvn = 0.0f;
            if (!do_surface) {
                hn = st.x; hun = st.y; hvn = st.z;
            } else if (info & CELL_ACTIVE) {
                const float rain = KIND == 1 ? s.rain_f * hz.w : s.rain_f;
                const float infil = KIND == 1 ? hz.y + (hz.x - hz.y) * __expf(-hz.z * wt) : a.infil_scalar;
                const CellNew u = cell_update(st, ci, &s_flux[tid * 3], dt, s.dtg_f, md, rain, infil);
                hn = u.h; hun = u.hu; hvn = u.hv;
                led[0] += u.rd * ci.x;
                led[1] += u.id * ci.x;
            }
            if (s.phases & FL_PHASE_CLAMP) clamp_velocity_exact(hn, hun, hvn, a.vmax);
            if (sent) send_state(x.exchange + (size_t)((base + k + 1) & 1u) * x.cells + c, hn, hun, hvn, base + k + 1);
            S.st[tid] = make_float4(hn, hun, hvn, st.w);
#pragma unroll
            for (int j = 0; j < 3; ++j) s_flux[tid * 3 + j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (KIND == 1 && do_surface) wt = wt + dt * (float)(hn > md);
            if (s.snap_slot >= 0) {
                const size_t o = (size_t)s.snap_slot * (size_t)a.C + (size_t)c;
                a.snap_h[o] = hn;
                a.snap_hu[o] = hun;
                a.snap_hv[o] = hvn;
            }
        }
#pragma unroll
        for (int j = 0; j < SURF_TERMS; ++j) {
            float y = led[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) y += __shfl_down_sync(0xffffffffu, y, o);
            if ((tid & 31) == 0) ff_accumulate(&total[j], y);
        }
    }
    // k steps were run: the states go where the next launch reads them
    if (c < a.C) {
        if (k > 0) (((first.parity ^ k) & 1) ? a.state1 : a.state0)[c] = S.st[tid];
        if (KIND == 1) a.wet[c] = wt;
    }
    if ((tid & 31) == 0) {
#pragma unroll
        for (int j = 0; j < SURF_TERMS; ++j) ledger[j] = total[j];
    }
}

// Global CFL minimum over all cells; the last block plans the step.
__global__ void __launch_bounds__(256) k_dt(const __grid_constant__ DtArgs a, int slot, int plan) {
    const float4 *__restrict__ st = a.run->parity ? a.state1 : a.state0;
    float best = CUDART_INF_F;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < a.C; c += gridDim.x * blockDim.x) {
        const float4 v = st[c];
        const float local = a.li ? cfl_local_li(v.x, a.char_len[c], a.cfl, a.g, a.md)
                                 : cfl_local(v.x, v.y, v.z, a.char_len[c], a.cfl, a.g, a.md);
        if (isfinite(local) && local < best) best = local;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = fminf(best, __shfl_xor_sync(0xffffffffu, best, o));
    __shared__ float wmin[32];
    __shared__ bool last;
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = wmin[0];
        for (int w = 1; w < (int)((blockDim.x + 31) >> 5); ++w) b = fminf(b, wmin[w]);
        a.partial[blockIdx.x] = b;
        __threadfence();
        const unsigned int done = atomicAdd(a.counter, 1u);
        last = (done == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    float b = CUDART_INF_F;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) b = fminf(b, ((volatile float *)a.partial)[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = fminf(b, __shfl_xor_sync(0xffffffffu, b, o));
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = wmin[0];
        for (int w = 1; w < (int)((blockDim.x + 31) >> 5); ++w) m = fminf(m, wmin[w]);
        if (a.dt_out) *a.dt_out = (m < CUDART_INF_F) ? (double)m : -1.0;
        if (plan) plan_step(a.run, a.snap_t, a.hy, &a.ctrl[slot], true, m, FL_PHASE_ALL);
        *a.counter = 0u;
    }
}

// Re-plan a step after fl_run changed the stop time (single thread).
__global__ void k_replan(RunCtrl *run, double *snap_t, HyetoView hy, StepCtrl *ctrl, int slot) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && !ctrl[slot].active) {
        plan_step(run, snap_t, hy, &ctrl[slot], false, 0.0f, FL_PHASE_ALL);
    }
}

// Non-finite depth check of the latest state (the reference checks h).
__global__ void k_finite(const float4 *state0, const float4 *state1, RunCtrl *run, int32_t C) {
    const float4 *st = run->parity ? state1 : state0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < C; c += gridDim.x * blockDim.x) {
        if (!isfinite(st[c].x)) {
            if (atomicCAS(&run->error, 0, FL_E_NONFINITE) == 0) run->error_step = run->step;
            return;
        }
    }
}

// ---------------------------------------------------------------- I/O
// state[new] <- reference-order arrays (perm[new] = reference index)
__global__ void k_load_state(float4 *state, const float *h, const float *hu, const float *hv,
                             const float *bed, const int32_t *perm, int32_t C, int mask) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < C; c += gridDim.x * blockDim.x) {
        const int r = perm[c];
        float4 v = state[c];
        if (mask & 1) v.x = h[r];
        if (mask & 2) v.y = hu[r];
        if (mask & 4) v.z = hv[r];
        v.w = bed[c];
        state[c] = v;
    }
}

__global__ void k_store_state(const float4 *state, float *h, float *hu, float *hv, const int32_t *perm,
                              int32_t C) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < C; c += gridDim.x * blockDim.x) {
        const int r = perm[c];
        const float4 v = state[c];
        if (h) h[r] = v.x;
        if (hu) hu[r] = v.y;
        if (hv) hv[r] = v.z;
    }
}

__global__ void k_permute_f32(const float *src, float *dst, const int32_t *perm, int32_t C, int to_reference) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < C; c += gridDim.x * blockDim.x) {
        if (to_reference) dst[perm[c]] = src[c];
        else dst[c] = src[perm[c]];
    }
}

__global__ void k_f64_to_ff(const double *src, float2 *dst, int32_t n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double v = src[i];
        const float hi = (float)v;
        dst[i] = make_float2(hi, (float)(v - (double)hi));
    }
}

__global__ void k_ff_to_f64(const float2 *src, double *dst, int32_t n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        dst[i] = (double)src[i].x + (double)src[i].y;
    }
}

__global__ void k_f64_to_ff_perm(const double *src, float2 *dst, const int32_t *perm, int32_t n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double v = src[perm[i]];
        const float hi = (float)v;
        dst[i] = make_float2(hi, (float)(v - (double)hi));
    }
}

__global__ void k_ff_to_f64_perm(const float2 *src, double *dst, const int32_t *perm, int32_t n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        dst[perm[i]] = (double)src[i].x + (double)src[i].y;
    }
}

// Link flows between the reference's link order (host side) and the
// solver's (perm[new] = reference link).
__global__ void k_f64_to_f32_perm(const double *src, float *dst, const int32_t *perm, int32_t n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = (float)src[perm[i]];
}

__global__ void k_f32_to_f64_perm(const float *src, double *dst, const int32_t *perm, int32_t n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[perm[i]] = (double)src[i];
}

// Current surface volume sum(h * area) and node volume (float64 partials).
// Each of the VOL_BLOCKS blocks covers a fixed set of cells and nodes and
// writes its partial pair; the host adds the pairs in block order, so the
// result does not depend on scheduling.
__global__ void __launch_bounds__(256) k_volumes(const float4 *state0, const float4 *state1, const float4 *cinfo,
                                                 const float2 *V, RunCtrl *run, int32_t C, int32_t N, double *part) {
    __shared__ double red[8][2];
    const float4 *st = run->parity ? state1 : state0;
    double vs = 0.0, vn = 0.0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < C; c += gridDim.x * blockDim.x)
        vs += (double)(st[c].x * cinfo[c].x);
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x)
        vn += (double)V[n].x + (double)V[n].y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        vs += __shfl_down_sync(0xffffffffu, vs, o);
        vn += __shfl_down_sync(0xffffffffu, vn, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5][0] = vs;
        red[threadIdx.x >> 5][1] = vn;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < 8; ++w) {
            a += red[w][0];
            b += red[w][1];
        }
        part[2 * blockIdx.x] = a;
        part[2 * blockIdx.x + 1] = b;
    }
}

}  // namespace fl

// Host launch wrappers (C++ linkage, used by fl_solver.cpp).
namespace fl {

// Launched as a programmatic dependent of the previous kernel in the stream
// (the drainage kernel before it triggers at its start), so its CTAs are
// scheduled and set up while that kernel finishes.
cudaError_t launch_surface(const SurfArgs &a, int kind, int slot, int plan_next, int grid, int smem_bytes,
                           cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, (unsigned)std::max(a.members, 1));
    cfg.blockDim = dim3(SURF_THREADS);
    cfg.dynamicSmemBytes = (size_t)smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void (*fn)(SurfArgs, int, int) = a.members > 1 ? (kind ? k_surface<1, true> : k_surface<0, true>)
                                                   : (kind ? k_surface<1, false> : k_surface<0, false>);
    return cudaLaunchKernelEx(&cfg, fn, a, slot, plan_next);
}

// The persistent grid of k_surface: every CTA slot of the device (never more
// CTAs than tiles), the last one the planner.  Tile t goes to CTA t mod
// (slots - 1), so the first CTAs take one tile more than the rest; CTAs are
// dispatched breadth-first over the SMs, so every SM carries the same number
// of tiles to within one CTA's share.  (Fewer CTAs with equal tile counts
// leave some SMs a CTA short: those SMs idle while the fully loaded ones
// finish.)  The assignment is the same on every launch, so each per-warp
// ledger slot sums the same values in the same order.
cudaError_t plan_surface_launch(SurfArgs &a, int kind, int device, int *grid, int *smem_bytes) {
    *smem_bytes = surface_smem_layout(a, kind);
    const void *fn = kind ? (const void *)k_surface<1, false> : (const void *)k_surface<0, false>;
    const void *fm = kind ? (const void *)k_surface<1, true> : (const void *)k_surface<0, true>;
    // the limit belongs to the function, not to this solver: always the
    // device's own, or a later solver with smaller tiles would lower it below
    // what an earlier one launches with
    int per_sm = 0, sms = 0, most = 0;
    cudaError_t e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fm, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, SURF_THREADS, (size_t)*smem_bytes);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int slots = std::max(1, per_sm * sms - 1);
    const int ctas = std::max(1, std::min(slots, a.n_tiles));
    *grid = ctas + 1;
    // the dependent may wait beside this grid while both fit twice over
    a.early = 2ll * *grid * std::max(a.members, 1) <= per_sm * sms ? 1 : 0;
    return cudaSuccess;
}

// Whether k_surface_run can run the mesh: every tile's CTA and the planner resident
// at once (on 152 SMs up to 607 tiles, 155,000 cells), and a CTA per tile of
// k_surface's grid too.  The ledger has a slot per warp of that grid, and a single
// step adds a CTA's tiles up before its slot: with fewer CTAs than tiles (k_surface
// keeps two stages in shared memory, so wide halos cost it a CTA an SM that the run
// kernel still has) the run kernel would have slots that do not exist.
// *smem_bytes 0: it cannot.  serial_words: the zeroed words of RunArgs::serial.
cudaError_t plan_surface_run(const SurfArgs &a, int kind, int surf_grid, int device, int *smem_bytes, size_t *serial_words) {
    const void *fn = kind ? (const void *)k_surface_run<1> : (const void *)k_surface_run<0>;
    *smem_bytes = 0;
    *serial_words = (size_t)(a.n_tiles + 1) * SYNC_STRIDE;
    if (a.n_tiles + 1 != surf_grid) return cudaSuccess;
    return run_fits(fn, a.n_tiles + 1, a.off_stage + a.stage_bytes, device, smem_bytes);
}

cudaError_t launch_surface_run(const SurfArgs &a, int kind, const RunArgs &x, int slot, int steps, int smem_bytes,
                               cudaStream_t stream) {
    return launch_run(kind ? k_surface_run<1> : k_surface_run<0>, a, x, slot, steps, a.n_tiles + 1, smem_bytes, stream);
}

int surface_warps(int grid) { return grid * (TILE / 32); }

cudaError_t launch_dt(const DtArgs &a, int blocks, int slot, int plan, cudaStream_t stream) {
    k_dt<<<blocks, 256, 0, stream>>>(a, slot, plan);
    return cudaGetLastError();
}

cudaError_t launch_replan(RunCtrl *run, double *snap_t, HyetoView hy, StepCtrl *ctrl, int slot, cudaStream_t stream) {
    k_replan<<<1, 32, 0, stream>>>(run, snap_t, hy, ctrl, slot);
    return cudaGetLastError();
}

// Grid of the grid-stride helper kernels below: enough 256-thread blocks for
// n elements, at most `per_sm` blocks per SM of the current device.
static int helper_grid(int64_t n, int per_sm) {
    static int sms[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (sms[dev] == 0 && cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        sms[dev] = 1;
    const int64_t want = std::max<int64_t>(1, (n + 255) / 256);
    return (int)std::min<int64_t>(want, (int64_t)std::max(sms[dev], 1) * per_sm);
}

cudaError_t launch_finite(const float4 *s0, const float4 *s1, RunCtrl *run, int32_t C, cudaStream_t stream) {
    k_finite<<<helper_grid(C, 4), 256, 0, stream>>>(s0, s1, run, C);
    return cudaGetLastError();
}

cudaError_t launch_load_state(float4 *state, const float *h, const float *hu, const float *hv, const float *bed,
                              const int32_t *perm, int32_t C, int mask, cudaStream_t stream) {
    k_load_state<<<helper_grid(C, 4), 256, 0, stream>>>(state, h, hu, hv, bed, perm, C, mask);
    return cudaGetLastError();
}

cudaError_t launch_store_state(const float4 *state, float *h, float *hu, float *hv, const int32_t *perm, int32_t C,
                               cudaStream_t stream) {
    k_store_state<<<helper_grid(C, 4), 256, 0, stream>>>(state, h, hu, hv, perm, C);
    return cudaGetLastError();
}

cudaError_t launch_permute_f32(const float *src, float *dst, const int32_t *perm, int32_t C, int to_reference,
                               cudaStream_t stream) {
    k_permute_f32<<<helper_grid(C, 4), 256, 0, stream>>>(src, dst, perm, C, to_reference);
    return cudaGetLastError();
}

cudaError_t launch_f64_to_ff(const double *src, float2 *dst, int32_t n, cudaStream_t stream) {
    k_f64_to_ff<<<helper_grid(n, 2), 256, 0, stream>>>(src, dst, n);
    return cudaGetLastError();
}

cudaError_t launch_ff_to_f64(const float2 *src, double *dst, int32_t n, cudaStream_t stream) {
    k_ff_to_f64<<<helper_grid(n, 2), 256, 0, stream>>>(src, dst, n);
    return cudaGetLastError();
}

cudaError_t launch_f64_to_ff_perm(const double *src, float2 *dst, const int32_t *perm, int32_t n, cudaStream_t stream) {
    k_f64_to_ff_perm<<<helper_grid(n, 2), 256, 0, stream>>>(src, dst, perm, n);
    return cudaGetLastError();
}

cudaError_t launch_ff_to_f64_perm(const float2 *src, double *dst, const int32_t *perm, int32_t n, cudaStream_t stream) {
    k_ff_to_f64_perm<<<helper_grid(n, 2), 256, 0, stream>>>(src, dst, perm, n);
    return cudaGetLastError();
}

cudaError_t launch_f64_to_f32_perm(const double *src, float *dst, const int32_t *perm, int32_t n, cudaStream_t stream) {
    k_f64_to_f32_perm<<<helper_grid(n, 2), 256, 0, stream>>>(src, dst, perm, n);
    return cudaGetLastError();
}

cudaError_t launch_f32_to_f64_perm(const float *src, double *dst, const int32_t *perm, int32_t n, cudaStream_t stream) {
    k_f32_to_f64_perm<<<helper_grid(n, 2), 256, 0, stream>>>(src, dst, perm, n);
    return cudaGetLastError();
}

cudaError_t launch_volumes(const float4 *s0, const float4 *s1, const float4 *cinfo, const float2 *V, RunCtrl *run,
                           int32_t C, int32_t N, double *out2, cudaStream_t stream) {
    k_volumes<<<VOL_BLOCKS, 256, 0, stream>>>(s0, s1, cinfo, V, run, C, N, out2);
    return cudaGetLastError();
}

}  // namespace fl
