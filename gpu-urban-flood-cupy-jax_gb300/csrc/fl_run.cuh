// Runs of the surface alone in one cooperative launch between CFL evaluations, a
// CTA a tile (k_surface_run, k_li_run): the exchange between tiles and the
// planning that both share.
//
// After a step a CTA sends the states of the cells that other tiles read, each
// with its step's serial number in one 16-byte store, and polls its halo cells for
// theirs: one L2 round trip, no fence.  The exchange has two buffers in turn; a
// tile's step k + 2 overwrites what its step k sent, and starts after its
// neighbours' step k + 1, which read that (halos are mutual).
//
// Every CTA plans for itself: its ninth warp advances a copy of the run control by
// plan_step during the step before (the records depend on times alone, so all CTAs
// get the same ones), and the last CTA, which has no tile, writes the run control's
// end back when every other CTA has copied its start.  (One planner for all put two
// more L2 round trips across the dies into every step: 4.9 instead of 3.0 us on
// 20,000 cells.)
//
// A step that checks for non-finite depths ends the run as a launch a step does, the
// step after it still done: each CTA counts its finished check, and the record of
// the step after next is planned when all have (a step later, so the wait is rarely
// one), on the first failed check by then -- the same in every CTA.
//
// Serial numbers: SYNC_STRIDE words a tile, then the last CTA's.  All of them hold
// the same number between launches (each CTA adds `steps`, also when the run ends
// early or a wait gives up), so nothing has to be reset.  Co-residency comes from
// the cooperative launch; every wait is bounded.
#pragma once

#include "fl_device.cuh"

namespace fl {

constexpr uint64_t RUN_WAIT_NS = 1000000000ull;  // 1 s per wait on another tile
constexpr int SYNC_STRIDE = 8;      // words: a sector each
constexpr int RUN_THREADS = TILE + 32;


// Bounded poll: *p has reached v (serial numbers; they may wrap).
__device__ __forceinline__ bool poll_reached(const uint32_t *p, uint32_t v, uint64_t limit_ns = RUN_WAIT_NS) {
    uint64_t t0 = 0;
    for (int i = 0;; ++i) {
        uint32_t x;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
        if ((int32_t)(x - v) >= 0) return true;
        if ((i & 63) == 63) {
            if (t0 == 0) t0 = global_ns();
            else if (global_ns() - t0 > limit_ns) return false;
        }
    }
}

__device__ __forceinline__ void publish(uint32_t *p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// A state and the serial number of its step, as one 16-byte access each way.
__device__ __forceinline__ void send_state(float4 *p, float h, float hu, float hv, uint32_t serial) {
    const uint64_t lo = (uint64_t)__float_as_uint(h) | (uint64_t)__float_as_uint(hu) << 32;
    const uint64_t hi = (uint64_t)__float_as_uint(hv) | (uint64_t)serial << 32;
    asm volatile(
        "{\n"
        ".reg .b128 t;\n"
        "mov.b128 t, {%1, %2};\n"
        "st.relaxed.gpu.global.b128 [%0], t;\n"
        "}\n" ::"l"(p), "l"(lo), "l"(hi)
        : "memory");
}

// Bounded poll for the state with this serial number.
__device__ __forceinline__ bool receive_state(const float4 *p, uint32_t serial, float4 &v, uint64_t limit_ns = RUN_WAIT_NS) {
    uint64_t t0 = 0;
    for (int i = 0;; ++i) {
        uint64_t lo, hi;
        asm volatile(
            "{\n"
            ".reg .b128 t;\n"
            "ld.relaxed.gpu.global.b128 t, [%2];\n"
            "mov.b128 {%0, %1}, t;\n"
            "}\n"
            : "=l"(lo), "=l"(hi)
            : "l"(p)
            : "memory");
        if ((uint32_t)(hi >> 32) == serial) {
            v.x = __uint_as_float((uint32_t)lo);
            v.y = __uint_as_float((uint32_t)(lo >> 32));
            v.z = __uint_as_float((uint32_t)hi);
            return true;
        }
        if ((i & 63) == 63) {
            if (t0 == 0) t0 = global_ns();
            else if (global_ns() - t0 > limit_ns) return false;
        }
    }
}

// A thread found a non-finite depth in a step's finite check.
__device__ __forceinline__ void run_non_finite(RunCtrl *run, int64_t step) {
    atomicMax((unsigned long long *)&run->first_bad, ~(unsigned long long)step);
    atomicCAS(&run->error, 0, FL_E_NONFINITE);
}

// Bounded wait until all tiles' checks up to `step` are finished (`count` in all); a
// failed one among them goes into the run control that plans (a later step's, which
// a tile that is ahead may have recorded, does not: some CTAs would see it, others not).
__device__ __forceinline__ bool run_checked(RunCtrl *run, uint32_t count, int64_t step, RunCtrl *s_run) {
    if (!poll_reached(&run->checks, count)) return false;
    unsigned long long bad;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(bad) : "l"(&run->first_bad) : "memory");
    if (bad >= ~(unsigned long long)step) s_run->error = FL_E_NONFINITE;
    return true;
}

__device__ __forceinline__ bool run_all(bool p) {
    uint32_t r;
    asm volatile(
        "{\n"
        ".reg .pred pi, po;\n"
        "setp.ne.u32 pi, %1, 0;\n"
        "bar.red.and.pred po, 2, %2, pi;\n"
        "selp.u32 %0, 1, 0, po;\n"
        "}\n"
        : "=r"(r)
        : "r"((uint32_t)p), "n"(RUN_THREADS)
        : "memory");
    return r != 0;
}

// The CTA without a tile: the run control after the last step, written back when
// every tile's CTA has read its start (their serial numbers say so).
__device__ __forceinline__ void run_last_cta(RunCtrl *run, StepCtrl *ctrl, double *snap_t, const HyetoView &hy, const RunArgs &x,
                                             int n_tiles, uint32_t base, int steps, const StepCtrl &first, RunCtrl *s_run,
                                             StepCtrl *s_rec) {
    const int tid = threadIdx.x;
    bool ok = true;
    if (tid == 0) {
        *s_run = *run;
        s_run->error = 0;  // (first is active; a tile that is ahead may have set it since)
        *s_rec = first;
        uint32_t count = s_run->checks_base;
        bool check = first.check_finite != 0, before = false;  // of the records k - 1 and k - 2
        int64_t at = first.step, at_before = 0;
        for (int k = 1; k < steps && s_rec->active && ok; ++k) {  // (as run_records)
            if (before) ok = run_checked(run, count += n_tiles, at_before, s_run);
            before = check;
            at_before = at;
            plan_step(s_run, snap_t, hy, s_rec, false, 0.0f, FL_PHASE_ALL);
            check = s_rec->check_finite != 0;
            at = s_rec->step;
        }
        if (before && s_rec->active) count += n_tiles;  // counted in the last step, which plans none
        s_run->checks_base = count;
    }
    for (int t = tid; t < n_tiles; t += RUN_THREADS) ok = ok && poll_reached(x.serial + (size_t)t * SYNC_STRIDE, base + steps);
    ok = __syncthreads_and(ok);
    if (tid == 0) {
        const int err = ok ? s_run->error : FL_E_TIMEOUT;
        if (err && atomicCAS(&run->error, 0, err) == 0) run->error_step = s_run->error ? s_run->error_step : first.step;
        run->t = s_run->t;
        run->next_snap_t = s_run->next_snap_t;
        run->step = s_run->step;
        run->last_dt = s_run->last_dt;
        run->cfl_reused = s_run->cfl_reused;
        run->parity = s_run->parity;
        run->snap_count = s_run->snap_count;
        run->checks_base = s_run->checks_base;
        if (!s_rec->active) ctrl[0] = ctrl[1] = *s_rec;
        publish(x.serial + (size_t)n_tiles * SYNC_STRIDE, base + steps);
    }
}

// A tile's ninth warp: the next step's record during each step.
__device__ __forceinline__ void run_records(bool ok, int steps, const HyetoView &hy, RunCtrl *run, int n_tiles, RunCtrl *s_run,
                                            StepCtrl *s_ctrl) {
    uint32_t count = s_run->checks_base;
    bool check = false;  // of the step before
    int64_t at = 0;
    for (int k = 0; k < steps; ++k) {
        if (!run_all(ok) || !s_ctrl[k & 1].active) break;  // (the CTA has finished step k - 1)
        if (threadIdx.x == TILE) {
            if (check) {
                count += n_tiles;
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&run->checks) : "memory");
            }
            if (k + 1 < steps) {
                if (check) ok = run_checked(run, count, at, s_run);
                check = s_ctrl[k & 1].check_finite != 0;
                at = s_ctrl[k & 1].step;
                plan_step(s_run, nullptr, hy, &s_ctrl[(k + 1) & 1], false, 0.0f, FL_PHASE_ALL);
            }
        }
        __syncwarp();
    }
}

// The tile's halo states at the start of step k into st[TILE ..]: from the state
// buffer at the launch's first step, then from what the other tiles sent (a halo
// cell's bed, the fourth word, stays).
__device__ __forceinline__ bool run_halo(bool ok, int k, const float4 *in, const RunArgs &x, uint32_t base, const int32_t *hs, int n,
                                         float4 *st) {
    if (k == 0) {
        for (int j = threadIdx.x; j < n && ok; j += TILE) st[TILE + j] = in[hs[j]];
    } else {
        const float4 *from = x.exchange + (size_t)((base + k) & 1u) * x.cells;
        for (int j = threadIdx.x; j < n && ok; j += TILE) {
            float4 v;
            ok = receive_state(from + hs[j], base + k, v);
            st[TILE + j].x = v.x;
            st[TILE + j].y = v.y;
            st[TILE + j].z = v.z;
        }
    }
    return ok;
}

// Host: *smem_bytes = bytes where `ctas` CTAs of a run kernel are resident at once.
inline cudaError_t run_fits(const void *fn, int ctas, int bytes, int device, int *smem_bytes) {
    int per_sm = 0, sms = 0, most = 0, coop = 0;
    cudaError_t e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaFuncAttributes at{};
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, fn);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)at.sharedSizeBytes);
    if (e != cudaSuccess || !coop || bytes > most - (int)at.sharedSizeBytes) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, RUN_THREADS, (size_t)bytes);
    if (e == cudaSuccess && ctas <= per_sm * sms) *smem_bytes = bytes;
    return e;
}

template <class Args>
inline cudaError_t launch_run(void (*fn)(Args, RunArgs, int, int), const Args &a, const RunArgs &x, int slot, int steps, int ctas,
                              int smem_bytes, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(RUN_THREADS);
    cfg.dynamicSmemBytes = (size_t)smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, a, x, slot, steps);
}

}  // namespace fl
