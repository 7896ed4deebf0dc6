// Batched-ensemble kernels for sm_103a.
//
// k_surface_batch: the persistent, warp-specialised surface kernel of
// k_surface (fl_surface.cu) over the tiles of every active scenario of a
// batch.  The planner's list maps a virtual tile index to (scenario, tile); a
// CTA's producer warp brings its virtual tiles into two stages (bulk async
// copies of the tile's states, cell info, Horton fields, wet time, running
// maximum depth, edge entries and halo list; then cp.async gathers of the halo
// states) and its compute warps evaluate them with the same tile_entry /
// cell_update / clamp code as the single-scenario kernel, with the scenario's
// own dt, rain and flags.  Per tile it stores the step's ledger terms and,
// when the scenario's next step evaluates the CFL dt, the minimum local dt of
// the tile's output state -- plain stores, reduced per scenario by the planner.
// A tile's warp partials are added up after the next tile's opening barrier,
// so a tile costs two barriers of the compute warps and none of the CTA.
//
// Planning.  A step that follows a CFL evaluation needs the step's minima:
// k_plan_batch, one CTA per scenario, reduces its tiles' ledger terms and CFL
// minima, plans its next step with plan_step (the single-scenario planner) and
// writes the scenario's entry of the next step's list.  It sits between two
// surface launches, so its length counts in full: the run record and the
// hyetograph are brought to shared memory in one level of loads (read field by
// field by the one planning thread they made it 12 us a step; 7 here), and no CTA
// waits for the others -- the surface CTAs add up the tile counts.
// Any other next step depends on the clock alone.  Where all scenarios evaluate on
// the same steps, CTAs at the end of the surface launch plan it meanwhile, a warp
// per scenario, and add up the previous step's ledger terms (lists and terms have
// two buffers); then only one step in a CFL interval has a planning launch (300 s of 16 scenarios,
// 1.64 M cells: 41.1 -> 38.0 ms; 90 s of six, 27,000 cells: 2.08 -> 1.59 ms).
// A scenario whose step checks for non-finite depths ends with that step if the
// check fails, so its next step is planned when the step is done: by the launch's
// last CTA, without a wait of any other.  (Where checks come every few steps, a
// planning launch a step is cheaper.)
//
// k_cfl_batch: the CFL minima of every tile's initial state (before step 0).
#include "fl_batch.cuh"
#include "fl_device.cuh"

namespace fl {

constexpr uint64_t BATCH_WAIT_NS = 1000000000ull;  // 1 s per wait on a tile copy

__device__ __forceinline__ int find_entry(const int32_t *prefix, int n, int v) {
    int lo = 0, hi = n;  // prefix[lo] <= v < prefix[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] <= v) lo = mid; else hi = mid;
    }
    return lo;
}

template <int T>
struct BStage {
    float4 *st;     // [T + h_cap]
    float4 *ci;     // [T]
    float4 *hz;     // [T] (kind 1)
    float *wt;      // [T] (kind 1)
    float *hm;      // [T]
    float4 *en;     // [e_cap]
    int32_t *hs;    // [h_cap]
};

template <int T>
__device__ __forceinline__ BStage<T> bstage_at(const BatchArgs &a, unsigned char *smem, int s) {
    unsigned char *b = smem + a.off_stage + s * a.stage_bytes;
    BStage<T> t;
    t.st = (float4 *)b;
    t.ci = (float4 *)(b + a.so_ci);
    t.hz = (float4 *)(b + a.so_hz);
    t.wt = (float *)(b + a.so_wt);
    t.hm = (float *)(b + a.so_hm);
    t.en = (float4 *)(b + a.so_en);
    t.hs = (int32_t *)(b + a.so_hs);
    return t;
}

// Issue the bulk copies of tile t (scenario entry E) into a stage (one
// thread); the expected byte count is the sum of exactly the copies issued.
template <int KIND, int T>
__device__ __forceinline__ void issue_btile(const BatchArgs &a, const BatchEntry &E, int t, const int4 ti,
                                            const BStage<T> &S, uint32_t bar) {
    const float4 *in = (E.flags & BF_PARITY) ? a.state1 : a.state0;
    const uint32_t ent_bytes = (uint32_t)ti.y * 16u;
    const uint32_t halo_bytes = (uint32_t)((ti.w + 3) & ~3) * 4u;
    uint32_t bytes = T * 16u * 2u + T * 4u + ent_bytes + halo_bytes;
    if (KIND == 1) bytes += T * 16u + T * 4u;
    mbar_arrive_expect_tx(bar, bytes);
    const size_t c0 = (size_t)t * T;
    bulk_copy_g2s(smem_addr(S.st), in + c0, T * 16u, bar);
    bulk_copy_g2s(smem_addr(S.ci), a.cinfo + c0, T * 16u, bar);
    bulk_copy_g2s(smem_addr(S.hm), a.hmax + c0, T * 4u, bar);
    if (KIND == 1) {
        bulk_copy_g2s(smem_addr(S.hz), a.horton + c0, T * 16u, bar);
        bulk_copy_g2s(smem_addr(S.wt), a.wet + c0, T * 4u, bar);
    }
    if (ent_bytes) bulk_copy_g2s(smem_addr(S.en), a.ent + ti.x, ent_bytes, bar);
    if (halo_bytes) bulk_copy_g2s(smem_addr(S.hs), a.halo_src + ti.z, halo_bytes, bar);
}

// Named barrier and barrier-reduction among the T compute threads (id 1).
template <int T>
__device__ __forceinline__ void batch_sync() {
    asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory");
}

template <int T>
__device__ __forceinline__ bool batch_all(bool p) {
    uint32_t r;
    asm volatile(
        "{\n"
        ".reg .pred pi, po;\n"
        "setp.ne.u32 pi, %1, 0;\n"
        "bar.red.and.pred po, 1, %2, pi;\n"
        "selp.u32 %0, 1, 0, po;\n"
        "}\n"
        : "=r"(r)
        : "r"((uint32_t)p), "n"(T)
        : "memory");
    return r != 0;
}

// A scenario's entry of a list, from its planned step.
__device__ __forceinline__ void list_entry(const PlanArgs &a, int b, BatchList *list, const StepCtrl &nx, int cfl_interval) {
    const int t0 = a.scen_tile0[b];
    list->tiles[b] = nx.active ? a.scen_tile0[b + 1] - t0 : 0;
    if (nx.active) {
        BatchEntry e;
        e.dt = nx.dt_f;
        e.dtg = nx.dtg_f;
        e.rain = nx.rain_f;
        e.infil = a.scen_infil[b];
        e.scen = b;
        const bool cfl_next = step_mod(nx.step + 1, cfl_interval) == 0;
        e.flags = (nx.parity ? BF_PARITY : 0) | (cfl_next ? BF_CFL : 0) | (nx.check_finite ? BF_FINITE : 0) |
                  (nx.phases << BF_PHASE_SHIFT) | ((nx.snap_slot + 1) << BF_SNAP_SHIFT);
        e.tile0 = t0;
        e.cells = a.scen_cells[b];
        list->e[b] = e;
    } else {
        list->e[b].flags = 0;
    }
}

// One warp, beside the surface CTAs of the step in `slot`: scenario b's ledger
// terms of the step before (k_plan_batch's sums, its four warps one after the
// other) and its next step's record and list entry.  s_run: a run record and a
// step record of shared memory.
constexpr int PLAN_SMEM = 384;
static_assert(sizeof(RunCtrl) % 8 == 0 && sizeof(RunCtrl) + sizeof(StepCtrl) <= PLAN_SMEM, "a warp's records in shared memory");

// A scenario whose step checks for non-finite depths is left to plan_checked, when
// the step is done (CHECKED: its record has been written by other SMs meanwhile).
// Its flag is loaded with the rest, not in front of it, and the two are separate
// code: on small batches this planner is the step.
template <bool CHECKED>
__device__ __noinline__ void plan_ahead(const PlanArgs &a, int b, int lane, int slot, int mode, RunCtrl *s_run) {
    StepCtrl *rec = &a.ctrl[2 * b + (slot ^ 1)], *s_next = (StepCtrl *)(s_run + 1);
    RunCtrl *run = &a.run[b];
    const int flags = a.list[slot].e[b].flags, t0 = a.scen_tile0[b], t1 = a.scen_tile0[b + 1];
    for (int i = lane; i < (int)(sizeof(RunCtrl) / 4); i += 32)
        ((uint32_t *)s_run)[i] = CHECKED ? __ldcg((const uint32_t *)run + i) : ((const uint32_t *)run)[i];
    const bool had_step = rec->active != 0;  // (the record of the step before, overwritten below)
    if (((flags & BF_FINITE) != 0 && (mode & BP_NEXT)) != CHECKED) return;
    if (mode & BP_LEDGER) {
        const float4 *led = (const float4 *)a.tile_led + (size_t)(slot ^ 1) * a.n_tiles;
        float sum[SURF_TERMS] = {0.0f, 0.0f, 0.0f, 0.0f};
        float l[4][SURF_TERMS];
#pragma unroll
        for (int w = 0; w < 4; ++w)
#pragma unroll
            for (int j = 0; j < SURF_TERMS; ++j) l[w][j] = 0.0f;
        for (int t = t0 + lane; t < t1; t += 128) {
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                if (t + 32 * w >= t1) break;
                const float4 v = led[t + 32 * w];
                l[w][0] += v.x;
                l[w][1] += v.y;
                l[w][2] += v.z;
                l[w][3] += v.w;
            }
        }
        __syncwarp();
#pragma unroll
        for (int w = 0; w < 4; ++w)
#pragma unroll
            for (int j = 0; j < SURF_TERMS; ++j) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) l[w][j] += __shfl_xor_sync(0xffffffffu, l[w][j], o);
                sum[j] = w == 0 ? l[w][j] : sum[j] + l[w][j];
            }
        if (had_step) {
#pragma unroll
            for (int j = 0; j < SURF_TERMS; ++j)
                if (lane == j) ff_accumulate(&a.ledger[b * SURF_TERMS + j], sum[j]);
        }
    }
    __syncwarp();
    if (!(mode & BP_NEXT)) return;
    if (lane == 0) {
        const int before = s_run->error;
        plan_step(s_run, a.snap_t + (size_t)b * a.max_snaps, a.hy[b], s_next, false, CUDART_INF_F, FL_PHASE_SURFACE | FL_PHASE_CLAMP);
        list_entry(a, b, a.list + (slot ^ 1), *s_next, s_run->cfl_interval);
        *rec = *s_next;
        if (s_run->error != before && atomicCAS(&run->error, 0, s_run->error) == 0) run->error_step = s_run->error_step;
        run->t = s_run->t;
        run->next_snap_t = s_run->next_snap_t;
        run->last_dt = s_run->last_dt;
        run->step = s_run->step;
        run->cfl_reused = s_run->cfl_reused;
        run->parity = s_run->parity;
        run->snap_count = s_run->snap_count;
    }
}

// The compute threads of a CTA that is done with a step in which some scenario
// checks for non-finite depths: the last of the `ctas` CTAs with tiles plans for those
// scenarios.  smem: T / 32 records of PLAN_SMEM bytes and a word.
template <int T>
__device__ __noinline__ void plan_checked(const PlanArgs &a, int ctas, int slot, int mode, unsigned char *smem) {
    volatile uint32_t *s_last = (volatile uint32_t *)(smem + T / 32 * PLAN_SMEM);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        __threadfence();  // (this CTA's errors, ordered by the barrier before the call)
        const bool last = atomicAdd(a.arrived, 1u) == (uint32_t)ctas - 1;
        __threadfence();
        if (last) *a.arrived = 0u;
        *s_last = last;
    }
    batch_sync<T>();
    if (!*s_last) return;
    for (int b = warp; b < a.n; b += T / 32) {
        plan_ahead<true>(a, b, lane, slot, mode, (RunCtrl *)(smem + warp * PLAN_SMEM));
        __syncwarp();
    }
}

// Four CTAs of 256-cell tiles an SM (seven of 128): 56 registers.
template <int KIND, int T>
__global__ void __launch_bounds__(T + 32, T == 256 ? 4 : 7) k_surface_batch(const __grid_constant__ BatchArgs a, const __grid_constant__ PlanArgs p,
                                                                            int slot, int mode) {
    constexpr int W = T / 32;
    extern __shared__ __align__(128) unsigned char smem[];
    float4 *s_flux = (float4 *)smem;  // [T * 3]
    uint64_t *s_bar = (uint64_t *)(smem + a.off_bar);   // full[2], halo[2], empty[2]
    int4 *s_info = (int4 *)(smem + a.off_bar + 48);
    int *s_kt = (int *)(smem + a.off_bar + 80);         // [2][2] list entry and tile of each stage
    float *s_red = (float *)(smem + a.off_bar + 96);    // [W][5] warp partials
    int32_t *s_prefix = (int32_t *)(smem + a.off_list);
    BatchEntry *s_ent = (BatchEntry *)(smem + a.off_list + MAX_SCEN * 4 + 16);
    const int tid = threadIdx.x;
    if ((int)blockIdx.x >= a.ctas) {
        pdl_wait();
        if (a.early) pdl_launch_dependents();
        const int b = ((int)blockIdx.x - a.ctas) * W + (tid >> 5);
        if (tid < T && b < p.n) plan_ahead<false>(p, b, tid & 31, slot, mode, (RunCtrl *)(smem + (tid >> 5) * PLAN_SMEM));
        return;
    }
    const uint32_t bar_base = smem_addr(s_bar);
    if (tid < T) {
#pragma unroll
        for (int k = 0; k < 3; ++k) s_flux[tid * 3 + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (tid == 0) {
        for (int k = 0; k < 2; ++k) {
            mbar_init(bar_base + 8u * k, 1);
            mbar_init(bar_base + 16u + 8u * k, 32);
            mbar_init(bar_base + 32u + 8u * k, W);
        }
        mbar_fence_init();
    }
    pdl_wait();  // the planner's list (its launch overlaps the set-up above)
    if (a.early) pdl_launch_dependents();
    const int n = a.n_scen;
    const BatchList *list = a.list + slot;
    float *tile_led = a.tile_led + (size_t)slot * a.n_tiles * SURF_TERMS;
    for (int i = tid; i < n; i += T + 32) s_ent[i] = list->e[i];
    if (tid < 32) {  // running sums of the tile counts (an inactive scenario's range is empty)
        constexpr int PER = MAX_SCEN / 32;
        int c[PER], sum = 0;
#pragma unroll
        for (int j = 0; j < PER; ++j) c[j] = tid * PER + j < n ? list->tiles[tid * PER + j] : 0;
#pragma unroll
        for (int j = 0; j < PER; ++j) sum += c[j];
        int before = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, before, o);
            if (tid >= o) before += x;
        }
        before -= sum;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            if (tid * PER + j <= n) s_prefix[tid * PER + j] = before;
            before += c[j];
        }
        if (tid == 31 && n == MAX_SCEN) s_prefix[n] = before;
    }
    __syncthreads();  // the last block-wide barrier: the roles split here
    const int total = s_prefix[n];
    const int G = a.ctas;
    const BStage<T> S0 = bstage_at<T>(a, smem, 0), S1 = bstage_at<T>(a, smem, 1);
    auto fail = [&]() {  // (one thread)
        for (int k = 0; k < n; ++k)
            if (atomicCAS(&a.run[k].error, 0, FL_E_TIMEOUT) == 0) a.run[k].error_step = p.ctrl[2 * k + slot].step;
    };

    if (tid >= T) {
        // ---------------------------------------------------------- producer
        const int lane = tid - T;
        bool failed = false;
        int i = 0;
        for (int v = blockIdx.x; v < total; v += G, ++i) {
            const int st = i & 1;
            const BStage<T> &S = st ? S1 : S0;
            const uint32_t full = bar_base + 8u * st;
            if (i >= 2) {  // the compute warps released this stage's previous tile
                bool ok = true;
                if (lane == 0) ok = mbar_wait_bounded(bar_base + 32u + 8u * st, ((i >> 1) - 1) & 1u, BATCH_WAIT_NS);
                if (!__shfl_sync(0xffffffffu, ok, 0)) {
                    failed = true;
                    break;
                }
            }
            if (lane == 0) {
                const int k = find_entry(s_prefix, n, v);
                const int t = s_ent[k].tile0 + (v - s_prefix[k]);
                const int4 ti = a.tile_info[t];
                s_kt[2 * st] = k;
                s_kt[2 * st + 1] = t;
                s_info[st] = ti;
                issue_btile<KIND, T>(a, s_ent[k], t, ti, S, full);
            }
            // every lane waits: each then reads the landed halo list itself
            const bool ok = mbar_wait_bounded(full, (i >> 1) & 1u, BATCH_WAIT_NS);
            if (!__all_sync(0xffffffffu, ok)) {
                // a copy is late: one more bounded wait so none lands after the CTA leaves
                (void)mbar_wait_bounded(full, (i >> 1) & 1u, BATCH_WAIT_NS);
                failed = true;
                break;
            }
            const float4 *in = (s_ent[s_kt[2 * st]].flags & BF_PARITY) ? a.state1 : a.state0;
            const int hc = s_info[st].w;
            for (int j = lane; j < hc; j += 32) cp_async16(smem_addr(&S.st[T + j]), in + S.hs[j]);
            cp_async_arrive_noinc(bar_base + 16u + 8u * st);
        }
        cp_async_wait_all();
        if (failed && lane == 0) fail();
        return;
    }

    // ------------------------------------------------------------- compute
    const float md = a.md;
    // whether some scenario checks for non-finite depths (while the first tile's copies are under way)
    bool check = false;
    if (mode & BP_NEXT)
        for (int k = tid; k < n; k += T) check = check || (s_ent[k].flags & BF_FINITE);
    const bool checked = (mode & BP_NEXT) && !batch_all<T>(!check);
    // the tile's ledger terms and CFL minimum from its warp partials (one thread)
    auto finish_tile = [&](int t, bool cfl) {
#pragma unroll
        for (int j = 0; j < SURF_TERMS; ++j) {
            float sum = 0.0f;
#pragma unroll
            for (int w = 0; w < W; ++w) sum += s_red[w * 5 + j];
            tile_led[(size_t)t * SURF_TERMS + j] = sum;
        }
        if (cfl) {
            float m = CUDART_INF_F;
#pragma unroll
            for (int w = 0; w < W; ++w) m = fminf(m, s_red[w * 5 + 4]);
            a.tile_min[t] = m;
        }
    };
    int i = 0, done_t = -1;
    bool done_cfl = false;
    for (int v = blockIdx.x; v < total; v += G, ++i) {
        const int st_i = i & 1;
        const BStage<T> &S = st_i ? S1 : S0;
        bool ok = true;
        if (tid == 0)
            ok = mbar_wait_bounded(bar_base + 8u * st_i, (i >> 1) & 1u, BATCH_WAIT_NS) &&
                 mbar_wait_bounded(bar_base + 16u + 8u * st_i, (i >> 1) & 1u, BATCH_WAIT_NS);
        if (!batch_all<T>(ok)) {  // also: every warp's partials of the previous tile are in place
            if (tid == 0) fail();
            done_t = -1;
            break;  // the producer waits out its own copies
        }
        if (tid == 0 && done_t >= 0) finish_tile(done_t, done_cfl);
        const BatchEntry &E = s_ent[s_kt[2 * st_i]];
        const int t = s_kt[2 * st_i + 1];
        const int flags = E.flags;
        const float dt = E.dt;
        const int phases = (flags >> BF_PHASE_SHIFT) & 7;
        const bool do_surface = (phases & FL_PHASE_SURFACE) != 0;
        float led[SURF_TERMS] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (do_surface) {
            const int n_e = s_info[st_i].y;
#pragma unroll 1
            for (int e = tid; e < n_e; e += T) tile_entry(S.en[e], S.st, s_flux, a.g, a.half_g, md, a.stage, dt, led[2], led[3]);
        }
        batch_sync<T>();  // phase 2's slots are complete

        // phase 3: the cell update
        const int c_local = (t - E.tile0) * T + tid;
        const size_t c = (size_t)t * T + tid;
        float cmin = CUDART_INF_F;
        if (c_local < E.cells) {
            const float4 st = S.st[tid];
            const float4 ci = S.ci[tid];
            const uint32_t info = __float_as_uint(ci.z);
            if ((flags & BF_FINITE) && !isfinite(st.x)) {
                if (atomicCAS(&a.run[E.scen].error, 0, FL_E_NONFINITE) == 0) a.run[E.scen].error_step = p.ctrl[2 * E.scen + slot].step;
            }
            float wt = 0.0f;
            float4 hz = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
            if (KIND == 1) {
                wt = S.wt[tid];
                hz = S.hz[tid];
            }
            float hn = st.x, hun = st.y, hvn = st.z;
            if (do_surface) {
                if (info & CELL_ACTIVE) {
                    const float rain = KIND == 1 ? E.rain * hz.w : E.rain;
                    const float infil = KIND == 1 ? hz.y + (hz.x - hz.y) * __expf(-hz.z * wt) : E.infil;
                    const CellNew u = cell_update(st, ci, &s_flux[tid * 3], dt, E.dtg, md, rain, infil);
                    hn = u.h; hun = u.hu; hvn = u.hv;
                    led[0] += u.rd * ci.x;
                    led[1] += u.id * ci.x;
                } else {
                    hn = 0.0f; hun = 0.0f; hvn = 0.0f;
                }
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) s_flux[tid * 3 + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (phases & FL_PHASE_CLAMP) clamp_velocity_exact(hn, hun, hvn, a.vmax);
            (flags & BF_PARITY ? a.state0 : a.state1)[c] = make_float4(hn, hun, hvn, st.w);
            if (KIND == 1 && do_surface) a.wet[c] = wt + dt * (float)(hn > md);
            const float hm = fmax32(S.hm[tid], hn);
            const int snap = (flags >> BF_SNAP_SHIFT) - 1;
            if (snap >= 0) {
                const size_t o = (size_t)a.snap_base[E.scen] + (size_t)snap * (size_t)E.cells + (size_t)c_local;
                a.snap_h[o] = hn;
                a.snap_hmax[o] = hm;
                a.snap_hu[o] = hun;
                a.snap_hv[o] = hvn;
                a.hmax[c] = 0.0f;
            } else {
                a.hmax[c] = hm;
            }
            if (flags & BF_CFL) {
                const float local = cfl_local(hn, hun, hvn, a.char_len[c], a.cfl, a.g, md);
                if (isfinite(local)) cmin = local;
            }
        }
        // the warp's partials; its lanes are done with the stage
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(bar_base + 32u + 8u * st_i);
#pragma unroll
        for (int j = 0; j < SURF_TERMS; ++j) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) led[j] += __shfl_down_sync(0xffffffffu, led[j], o);
        }
        if (flags & BF_CFL) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) cmin = fminf(cmin, __shfl_down_sync(0xffffffffu, cmin, o));
        }
        if ((tid & 31) == 0) {
#pragma unroll
            for (int j = 0; j < SURF_TERMS; ++j) s_red[(tid >> 5) * 5 + j] = led[j];
            s_red[(tid >> 5) * 5 + 4] = cmin;
        }
        done_t = t;
        done_cfl = (flags & BF_CFL) != 0;
    }
    if (done_t >= 0 || checked) {
        batch_sync<T>();
        if (tid == 0 && done_t >= 0) finish_tile(done_t, done_cfl);
    }
    if (checked) plan_checked<T>(p, G, slot, mode, smem);
}

// CFL minima of every tile's state before the first step (all scenarios'
// states in state0).
template <int T>
__global__ void __launch_bounds__(T) k_cfl_batch(const float4 *state0, const float *char_len, const int32_t *tile_valid,
                                                 float *tile_min, float cfl, float g, float md) {
    const int t = blockIdx.x;
    const int tid = threadIdx.x;
    float m = CUDART_INF_F;
    if (tid < tile_valid[t]) {
        const size_t c = (size_t)t * T + tid;
        const float4 v = state0[c];
        const float local = cfl_local(v.x, v.y, v.z, char_len[c], cfl, g, md);
        if (isfinite(local)) m = local;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float wmin[T / 32];
    if ((tid & 31) == 0) wmin[tid >> 5] = m;
    __syncthreads();
    if (tid == 0) {
        float b = wmin[0];
#pragma unroll
        for (int w = 1; w < T / 32; ++w) b = fminf(b, wmin[w]);
        tile_min[t] = b;
    }
}

// One CTA per scenario: fold the step's tile terms into the scenario's
// ledger, plan its next step and write its entry of the list.
constexpr int PLAN_HYETO = 128;  // hyetograph blocks held in shared memory

__global__ void __launch_bounds__(128) k_plan_batch(const __grid_constant__ PlanArgs a, int slot, int init) {
    __shared__ RunCtrl s_run;
    __shared__ StepCtrl s_next;
    __shared__ double s_hy[3][PLAN_HYETO];
    __shared__ float red[4][SURF_TERMS + 1];
    const int b = blockIdx.x;
    const int tid = threadIdx.x;
    const int t0 = a.scen_tile0[b], t1 = a.scen_tile0[b + 1];
    HyetoView hy = a.hy[b];
    if (hy.n <= PLAN_HYETO) {  // (inputs: not written by the step)
        if (tid < hy.n) {
            s_hy[0][tid] = hy.start_s[tid];
            s_hy[1][tid] = hy.end_s[tid];
            s_hy[2][tid] = hy.rate[tid];
        }
        hy.start_s = s_hy[0];
        hy.end_s = s_hy[1];
        hy.rate = s_hy[2];
    }
    pdl_wait();               // the step's surface kernel
    pdl_launch_dependents();  // the next one may set up meanwhile
    RunCtrl *run = &a.run[b];
    static_assert(sizeof(RunCtrl) % 4 == 0 && sizeof(RunCtrl) <= 128 * 4 && sizeof(StepCtrl) % 4 == 0 && sizeof(StepCtrl) <= 128 * 4,
                  "records are copied a word per thread");
    if (tid < (int)(sizeof(RunCtrl) / 4)) ((uint32_t *)&s_run)[tid] = ((const uint32_t *)run)[tid];
    const int cfl_interval = run->cfl_interval;
    const int cur_active = a.ctrl[2 * b + slot].active;
    const int64_t cur_step = a.ctrl[2 * b + slot].step;
    float m = CUDART_INF_F;
    float l[SURF_TERMS] = {0.0f, 0.0f, 0.0f, 0.0f};
    static_assert(SURF_TERMS == 4, "a tile's ledger terms are one float4");
    const float4 *led = (const float4 *)a.tile_led + (size_t)slot * a.n_tiles;
    for (int t = t0 + tid; t < t1; t += 128 * 4) {  // four tiles' loads in flight (whether or not the step uses them), added in order
        float4 v[4];
        float q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool in = t + u * 128 < t1;
            v[u] = in ? led[t + u * 128] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            q[u] = in ? a.tile_min[t + u * 128] : CUDART_INF_F;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (t + u * 128 >= t1) break;
            m = fminf(m, q[u]);
            l[0] += v[u].x;
            l[1] += v[u].y;
            l[2] += v[u].z;
            l[3] += v[u].w;
        }
    }
    const bool had_step = !init && cur_active;
    const bool cfl_done = init || (had_step && step_mod(cur_step + 1, cfl_interval) == 0);
    if (!cfl_done) m = CUDART_INF_F;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
#pragma unroll
        for (int j = 0; j < SURF_TERMS; ++j) l[j] += __shfl_xor_sync(0xffffffffu, l[j], o);
    }
    if ((tid & 31) == 0) {
#pragma unroll
        for (int j = 0; j < SURF_TERMS; ++j) red[tid >> 5][j] = l[j];
        red[tid >> 5][SURF_TERMS] = m;
    }
    __syncthreads();
    if (tid < SURF_TERMS && had_step)
        ff_accumulate(&a.ledger[b * SURF_TERMS + tid], red[0][tid] + red[1][tid] + red[2][tid] + red[3][tid]);
    if (tid == 32) {  // (a warp of its own: the ledger's round trip does not delay it)
        float mm = red[0][SURF_TERMS];
        for (int w = 1; w < 4; ++w) mm = fminf(mm, red[w][SURF_TERMS]);
        const bool eval = step_mod(s_run.step, cfl_interval) == 0;
        plan_step(&s_run, a.snap_t + (size_t)b * a.max_snaps, hy, &s_next, eval, mm, FL_PHASE_SURFACE | FL_PHASE_CLAMP);
        list_entry(a, b, a.list + (slot ^ 1), s_next, cfl_interval);
    }
    __syncthreads();
    if (tid < (int)(sizeof(RunCtrl) / 4)) ((uint32_t *)run)[tid] = ((const uint32_t *)&s_run)[tid];
    if (tid < (int)(sizeof(StepCtrl) / 4)) ((uint32_t *)&a.ctrl[2 * b + (slot ^ 1)])[tid] = ((const uint32_t *)&s_next)[tid];
}

template __global__ void k_surface_batch<0, 128>(const __grid_constant__ BatchArgs, const __grid_constant__ PlanArgs, int, int);
template __global__ void k_surface_batch<0, 256>(const __grid_constant__ BatchArgs, const __grid_constant__ PlanArgs, int, int);
template __global__ void k_surface_batch<1, 128>(const __grid_constant__ BatchArgs, const __grid_constant__ PlanArgs, int, int);
template __global__ void k_surface_batch<1, 256>(const __grid_constant__ BatchArgs, const __grid_constant__ PlanArgs, int, int);

static const void *surface_batch_fn(int kind, int tile) {
    if (kind) return tile == 128 ? (const void *)k_surface_batch<1, 128> : (const void *)k_surface_batch<1, 256>;
    return tile == 128 ? (const void *)k_surface_batch<0, 128> : (const void *)k_surface_batch<0, 256>;
}

cudaError_t batch_configure(int kind, int tile, int smem_bytes, int *per_sm) {
    const void *fn = surface_batch_fn(kind, tile);
    // the device's own limit: the attribute is the function's, shared by every batch
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, fn, tile + 32, (size_t)smem_bytes);
}

// Launch as a programmatic dependent of the previous kernel in the stream.
template <class Args, class... Rest>
static cudaError_t launch_dependent(void (*kernel)(Args, Rest...), int grid, int threads, int smem_bytes, cudaStream_t stream,
                                    const Args &a, Rest... rest) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a, rest...);
}

int batch_plan_ctas(int tile, int n) { return (n + tile / 32 - 1) / (tile / 32); }

cudaError_t launch_surface_batch(const BatchArgs &a, const PlanArgs &p, int kind, int slot, int mode, int smem_bytes,
                                 cudaStream_t stream) {
    void (*fn)(BatchArgs, PlanArgs, int, int) = a.tile == 128 ? (kind ? k_surface_batch<1, 128> : k_surface_batch<0, 128>)
                                                              : (kind ? k_surface_batch<1, 256> : k_surface_batch<0, 256>);
    return launch_dependent(fn, a.ctas + (mode ? batch_plan_ctas(a.tile, a.n_scen) : 0), a.tile + 32, smem_bytes, stream, a, p, slot,
                            mode);
}

cudaError_t launch_cfl_batch(const float4 *state0, const float *char_len, const int32_t *tile_valid, float *tile_min,
                             int tiles, int tile, float cfl, float g, float md, cudaStream_t stream) {
    if (tile == 128) k_cfl_batch<128><<<tiles, 128, 0, stream>>>(state0, char_len, tile_valid, tile_min, cfl, g, md);
    else k_cfl_batch<256><<<tiles, 256, 0, stream>>>(state0, char_len, tile_valid, tile_min, cfl, g, md);
    return cudaGetLastError();
}

cudaError_t launch_plan_batch(const PlanArgs &a, int slot, int init, cudaStream_t stream) {
    return launch_dependent(k_plan_batch, a.n, 128, 0, stream, a, slot, init);
}

}  // namespace fl
