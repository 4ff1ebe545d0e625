// A fast time step (steps >= 1 of configurations with a ring table) as ONE
// kernel, with no boundary kernel and no end-of-step election:
//   * every block first works out the PREVIOUS step's end (t, dt, stop flags)
//     from its wave-speed maximum, for itself, the same bits in every block;
//     block 0 records it for the next launch;
//   * interior warps march over rows 2..L-1 (lf_tma.cuh);
//   * ring warps compute the boundary ring at the same time, one lane per
//     cell: the new value a face reads next to the ring is recomputed from the
//     step's input state (fast_cell_alone: the interior warp's operations in
//     the same order, the same bits), so nothing waits for the interior.
// Before, a boundary kernel followed the interior: its hand-off, its cells'
// interpreted chains (8.2 us of a 36 us step at 1600 x 640), its last-block
// election and the controller stood between two interiors, 12 us of the step,
// and nearly all of the 11.8 us step at 100 x 40.
//
// Launch i of a sequence takes slot = i & 1: it reads ctl[slot] and writes
// ctl[slot ^ 1].  A stopped run's remaining launches copy the slot on.
// finish_steps_kernel ends a sequence: it works out the last step's
// controller, leaves the canonical DevState fields, slot 0 current and the
// wave-speed maxima zero.
#pragma once

#include <cuda_runtime.h>

#include "kernels.cuh"
#include "lf_tma.cuh"

namespace mpd {

using StepRun = StepHot::Run;

// One slot's controller and the wave-speed line as a warp's words: lane k the
// k-th 8-byte word of ctl[slot] (k < 8), lane 16 + k that of acc (k < 6).  Two
// requests to L2 for a whole block: with every thread of a launch loading the
// fields for itself, 444 blocks queued on the two lines and the median block
// began its march 4.5 us after the first could have (1600 x 640, B200).
struct StepWords {
    unsigned long long w;
    __device__ __forceinline__ void load(const StepHot *h, int slot, int lane) {
        const unsigned long long *c = reinterpret_cast<const unsigned long long *>(&h->ctl[slot]);
        const unsigned long long *a = reinterpret_cast<const unsigned long long *>(&h->acc);
        w = 0ull;
        if (lane < 7) w = __ldcg(c + lane);
        if (lane >= 16 && lane < 22) w = __ldcg(a + lane - 16);
    }
    __device__ __forceinline__ unsigned long long u(int k) const {
        return __shfl_sync(0xffffffffu, w, k);
    }
    __device__ __forceinline__ double d(int k) const {
        return __longlong_as_double((long long)u(k));
    }
    __device__ __forceinline__ StepCtl ctl() const {
        StepCtl c{};
        c.t = d(0);
        c.dt = d(1);
        c.dt_used = d(2);
        c.last_ws = d(3);
        c.step = (long long)u(4);
        const unsigned long long a = u(5), b = u(6);
        c.stepped = (int)(unsigned int)a;
        c.done = (int)(a >> 32);
        c.nonfinite = (int)(unsigned int)b;
        c.ws_valid = (int)(b >> 32);
        return c;
    }
    __device__ __forceinline__ unsigned long long ws(int k) const { return u(16 + k); }
    __device__ __forceinline__ unsigned int nf(int k) const {
        return (unsigned int)(u(19 + k / 2) >> (32 * (k & 1)));
    }
    __device__ __forceinline__ int wait_fail() const { return (int)(unsigned int)u(21); }
};
// The run parameters the same way: one request of one warp.
__device__ __forceinline__ StepRun step_run(const StepHot *h, int lane) {
    const unsigned long long *p = reinterpret_cast<const unsigned long long *>(&h->run);
    StepWords x;
    x.w = lane < 7 ? __ldcg(p + lane) : 0ull;
    StepRun r{};
    r.T = x.d(0);
    r.cfl = x.d(1);
    r.growth = x.d(2);
    r.dt_min = x.d(3);
    r.dt_max = x.d(4);
    r.max_steps = (long long)x.u(5);
    const unsigned long long f = x.u(6);
    r.run_mode = (int)(unsigned int)f;
    r.adaptive = (int)(f >> 32);
    return r;
}
static_assert(offsetof(StepRun, max_steps) == 40 && offsetof(StepRun, run_mode) == 48, "step_run");
static_assert(offsetof(StepCtl, step) == 32 && offsetof(StepCtl, nonfinite) == 48, "StepWords");
static_assert(offsetof(StepHot::Acc, nf) == 24 && offsetof(StepHot::Acc, wait_fail) == 40,
              "StepWords");

// The end of the step that led to c (step_controller's arithmetic): wave speed
// and non-finite flag, and in run mode the next dt and the stop condition.
// Every lane of a warp, the same values in each.
template <bool WANT_WS>
__device__ __forceinline__ StepCtl step_resolve(const Geo &g, const StepWords &x,
                                                const StepRun &r) {
    StepCtl c = x.ctl();
    const int k = (int)(c.step % 3);
    const double ws = WANT_WS ? __longlong_as_double((long long)x.ws(k)) : 0.0;
    const unsigned int f = x.nf(k);
    if (c.stepped) {
        if (WANT_WS) c.last_ws = ws;
        c.ws_valid = WANT_WS ? 1 : 0;
        c.nonfinite = (c.nonfinite || f || !isfinite(ws)) ? 1 : 0;
        if (r.run_mode) {
            double dtn = c.dt;
            if (r.adaptive)
                dtn = compute_dt_from_speed(ws, g.dz, g.dy, r.cfl, r.growth, r.dt_min, r.dt_max,
                                            c.dt);
            c.done = (c.nonfinite || !(c.t < r.T) || c.step >= r.max_steps) ? 1 : 0;
            if (c.t + dtn > r.T) dtn = r.T - c.t;
            c.dt = dtn;
        }
        c.stepped = 0;
    }
    if (x.wait_fail()) c.done = 1;
    return c;
}

static_assert(sizeof(RingSeg) % 16 == 0, "ring segments are copied as 16-byte words");

// A shared-memory double at a 32-bit shared address: explicitly the shared
// state space.  (An earlier form of the ring that picked operands between these
// slots and global arrays through one pointer at run time faulted.  The cause
// is not known; nothing is left of that form.)
__device__ __forceinline__ double lds_f64(uint32_t a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts_f64(uint32_t a, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// A lane's 8 primitive slots, a row of 32 doubles apart; a warp's two sets
// (the neighbour's, the cell's own) are 4 KB.
struct RingSlots {
    uint32_t a;
    __device__ __forceinline__ double get(int j) const { return lds_f64(a + 256u * (uint32_t)j); }
    __device__ __forceinline__ void set(int j, double v) const {
        sts_f64(a + 256u * (uint32_t)j, v);
    }
};

// Warps of a step; nring of them take 32 ring slots each.
//   alone (grids whose bands are a few rows, so that a ring cell costs as much
//   as several): ring warps take no rows; otherwise every warp has a band and
//   the ring warps' bands, the first nshort of each strip, are shorter by
//   MPD_RING_ROWS rows.
//   spread: one ring warp to a block, the last warp of blocks 0, 1, .. (four to
//   a block make that SM's load path the bottleneck, each of a wall warp's 40
//   loads touching 32 rows: 100 x 40 7.2 against 4.9 us a step, 1600 x 640 30.4
//   against 27.9).  Where the state is far larger than L2 the bands stay in
//   task order instead, ring warps first: neighbouring strips on neighbouring
//   warps share the sectors at their edges, and scattering the ring's bands
//   costs more (3000 x 1000: 87.5 against 84.4 us, 4096 x 1600: 192 against
//   170; the line lies between it and 2400 x 900: 59.4 against 61.6).
struct StepPlan {
    int nstrips = 0, nbands = 0, nring = 0, alone = 0, spread = 0, nshort = 0, blocks = 0;
};
#ifndef MPD_SPREAD_BYTES
#define MPD_SPREAD_BYTES (160ll << 20)
#endif

// Ring index of warp wib of a block (-1: none), and its interior task.
__host__ __device__ inline int step_ring(const StepPlan &p, int block, int wib) {
    const int i = p.spread ? block + p.blocks * (kTmaWarps - 1 - wib) : block * kTmaWarps + wib;
    return i < p.nring ? i : -1;
}
__host__ __device__ inline int step_task(const StepPlan &p, int block, int wib) {
    if (!p.spread) return block * kTmaWarps + wib;
    const int ring = step_ring(p, block, wib);
    if (ring >= 0) return p.alone ? -1 : ring;
    // the warps before this one that are no ring warps: those fill the last
    // warp of every block, then the one before it
    const int full = p.nring / p.blocks, rest = p.nring % p.blocks;
    const int before = block * (kTmaWarps - full) - (block < rest ? block : rest) + wib;
    return p.alone ? before : p.nring + before;
}

// What a ring warp's cells cost, in rows of a band.
#ifndef MPD_RING_ROWS
#define MPD_RING_ROWS 6
#endif
// Bands of at most this many rows: the ring in warps of its own.
constexpr int kRingAloneRows = 8;

// First row of band b (rows 2..L-1; bands of at least one row).
__host__ __device__ inline int step_band(const StepPlan &p, int L, int b) {
    const int rows = L - 2;
    if (p.nshort == 0) return 2 + (int)((long long)b * rows / p.nbands);
    // nshort bands of h - worth rows, the others of h
    const int worth = MPD_RING_ROWS;
    const long long total = rows + (long long)p.nshort * worth;
    const long long at = (long long)b * total / p.nbands;
    return 2 + (int)(at - (long long)(b < p.nshort ? b : p.nshort) * worth);
}

template <bool WANT_WS, bool AXIS>
__global__ void __launch_bounds__(32 * kTmaWarps, MPD_TMA_MINB)
    lf_step_kernel(Geo g, const __grid_constant__ CUtensorMap map0,
                   const __grid_constant__ CUtensorMap map1, double *buf0, double *buf1,
                   DevState *st, double dt_arg, int use_state_dt,
                   const __grid_constant__ RingTable ring, const __grid_constant__ StepPlan plan,
                   int slot, int parity) {
    extern __shared__ __align__(128) unsigned char step_smem_raw[];
    unsigned char *base = tma_smem_base(step_smem_raw);
    RingSeg *seg = reinterpret_cast<RingSeg *>(base + kTmaSmem - 128);
    const int wib = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int ring_i = step_ring(plan, blockIdx.x, wib);
    const int task = step_task(plan, blockIdx.x, wib);
    int strip = 0, l_begin = 2, l_end = 2;
    if (task >= 0 && task < plan.nstrips * plan.nbands) {
        strip = task % plan.nstrips;
        const int band = task / plan.nstrips;
        l_begin = step_band(plan, g.L, band);
        l_end = step_band(plan, g.L, band + 1);
    }
    const uint32_t bar0 =
        smem_addr(base + kTmaWarps * kTmaStages * kTmaRowBytes) + 8u * wib * kTmaStages;
    // While the previous kernel of the stream may still run: only this
    // block's shared memory, and what no kernel writes (the tensor maps, the
    // ring table, the run parameters).
    const bool band = l_begin < l_end;
    if (band && lane == 0) {
        tmap_prefetch(&map0);
        tmap_prefetch(&map1);
        for (int k = 0; k < kTmaStages; ++k) mbar_init(bar0 + 8u * k, 1);
        mbar_init_fence();
    }
    if ((plan.spread ? (int)blockIdx.x : (int)blockIdx.x * kTmaWarps) < plan.nring) {
        const int n = ring.nseg * (int)(sizeof(RingSeg) / sizeof(int4));
        const int4 *src = reinterpret_cast<const int4 *>(ring.seg);
        int4 *dst = reinterpret_cast<int4 *>(seg);
        for (int k = threadIdx.x; k < n; k += blockDim.x) dst[k] = src[k];
    }
    RingLane rl;
    const bool has_ring = ring_i >= 0;
    if (has_ring) rl.place(g, ring, ring_i * 32 + lane);
    __shared__ double s_dt;
    __shared__ long long s_step;
    __shared__ int s_done;
    StepRun run{};
    if (wib == 0) run = step_run(&st->hot, lane);
    pdl_wait();
    StepWords x;
    if (wib == 0) x.load(&st->hot, slot, lane);
    // parity: the step count's, where the host knows it (else -1; a wrong one
    // costs a second read).  Taken from the run parameters instead, so that one
    // graph serves runs from odd and even steps, the reads wait for that load:
    // 31.67 against 31.33 us a step at 1600 x 640.  The reads of spread ring warps then travel with the controller's (0.25 us a step at
    // 100 x 40); the bands' first rows asked for here too slowed the
    // controller's own reads by more than they gained.
    const bool early = parity >= 0 && plan.spread;
    if (early && has_ring) rl.load(g, parity == 1 ? buf1 : buf0);
    if (wib == 0) {
        const StepCtl c = step_resolve<WANT_WS>(g, x, run);
        const double dt0 = use_state_dt ? c.dt : dt_arg;
        if (lane == 0) {
            s_dt = dt0;
            s_step = c.step;
            s_done = c.done;
            if (blockIdx.x == 0) {
                StepCtl n = c;
                if (!c.done) {
                    n.t = c.t + dt0;
                    n.dt = n.dt_used = dt0;
                    n.step = c.step + 1;
                    n.stepped = 1;
                    const int clear = (int)((c.step + 2) % 3);
                    st->hot.acc.ws[clear] = 0ull;
                    st->hot.acc.nf[clear] = 0u;
                }
                st->hot.ctl[slot ^ 1] = n;
            }
        }
    }
    __syncthreads();
    const bool odd = (s_step & 1) != 0;
    if (s_done) return;
    const double dt = s_dt;
    const int acc = (int)((s_step + 1) % 3);
    unsigned long long ws_key = 0ull;
    unsigned int nf = 0u;
    if (has_ring) {
        if (!early || parity != (odd ? 1 : 0)) rl.load(g, odd ? buf1 : buf0);
        // the slots lie in this warp's row stages, free until its band begins
        const RingSlots nb = {smem_addr(base + wib * kTmaStages * kTmaRowBytes) + 8u * lane};
        const RingSlots cur = {nb.a + 2048u};
        if (rl.act) {
            double uf[8], r;
            ring_cell_new<AXIS>(g, ring, seg, rl, odd ? buf1 : buf0, dt, nb, cur, uf, r);
            double *u = odd ? buf0 : buf1;
            const size_t ix = g.ix(rl.l, rl.m);
#pragma unroll
            for (int k = 0; k < 8; ++k) u[(size_t)k * g.ps + ix] = uf[k];
            if (WANT_WS) {
                const double sp = fast_wave_speed(uf, r, rcp_nr(r), g.gamma);
                if (!isfinite(sp)) nf = 1u;
                const unsigned long long kk = max_key(sp, nf);
                ws_key = kk > ws_key ? kk : ws_key;
            }
        }
        // its generic accesses of the stages before the TMA's
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (band) {
        TmaWarp w;
        tma_warp_setup(w, g, strip, odd ? buf0 : buf1, st, nullptr, 0, dt, odd ? &map1 : &map0);
        w.stage = reinterpret_cast<double *>(base) + wib * kTmaStages * kTmaRow;
        w.bar0 = bar0;
        __syncwarp();
        uint32_t j = 0;
        const bool ok = tma_band_run<WANT_WS, false>(w, l_begin, l_end, j, ws_key, nf);
        if (!ok && lane == 0) {
            // a row never arrived: record the failure; later steps stop at it
            atomicExch(&st->wait_fail, 1);
            atomicExch(&st->hot.acc.wait_fail, 1);
            if (st->mirror) {
                st->mirror->wait_fail = 1;
                __threadfence_system();
            }
        }
    }
    pdl_trigger();
    if (WANT_WS) {
        unsigned long long key[1] = {ws_key};
        unsigned long long *dst[1] = {&st->hot.acc.ws[acc]};
        block_max_atomic<1>(key, nf, dst, &st->hot.acc.nf[acc]);
    }
}

// The end of a sequence of step launches, ctl[slot] current: one warp.  Leaves
// what step_controller leaves after a step.
template <bool WANT_WS>
__global__ void finish_steps_kernel(Geo g, DevState *st, int slot) {
    const StepRun run = step_run(&st->hot, threadIdx.x);
    pdl_wait();
    StepWords x;
    x.load(&st->hot, slot, threadIdx.x);
    const double conv_thr = __ldcg(&st->conv_thr);
    const int check_freq = __ldcg(&st->check_freq);
    const long long step0 = __ldcg(&st->step);
    const StepCtl c = step_resolve<WANT_WS>(g, x, run);
    const int wait_fail = x.wait_fail();
    if (threadIdx.x != 0) return;
    st->hot.ctl[0] = c;
    // the step has ended: no maximum is needed any more, and steps of another
    // kernel may come before the next of these, so all three start from zero
    for (int k = 0; k < 3; ++k) {
        st->hot.acc.ws[k] = 0ull;
        st->hot.acc.nf[k] = 0u;
    }
    if (c.step == step0) {
        if (run.run_mode && c.done) st->done = 1;
        return;
    }
    if (WANT_WS) st->last_ws = c.last_ws;
    st->ws_valid = c.ws_valid;
    st->nonfinite = c.nonfinite;
    st->t = c.t;
    st->dt_used = c.dt_used;
    st->step = c.step;
    st->resid_valid = 0;
    if (run.run_mode) {
        st->dt = c.dt;
        st->check_due =
            (conv_thr > 0.0 && check_freq > 0 && c.step % check_freq == 0) ? 1 : 0;
        st->done = c.done;
    }
    HostMirror *hm = run.run_mode ? nullptr : st->mirror;
    if (hm) {
        if (WANT_WS) hm->last_ws = c.last_ws;
        hm->ws_valid = c.ws_valid;
        hm->wait_fail = wait_fail;
        asm volatile("st.release.sys.b64 [%0], %1;" ::"l"(&hm->step), "l"(c.step) : "memory");
    }
}

inline int step_smem(int nseg) { return kTmaSmem + nseg * (int)sizeof(RingSeg); }

using StepKernel = void (*)(Geo, const CUtensorMap, const CUtensorMap, double *, double *,
                            DevState *, double, int, const RingTable, const StepPlan, int,
                            int);
inline StepKernel step_kernel(bool want_ws, const RingTable &t) {
    if (t.has_axis) return want_ws ? lf_step_kernel<true, true> : lf_step_kernel<false, true>;
    return want_ws ? lf_step_kernel<true, false> : lf_step_kernel<false, false>;
}

// One wave: strips x bands and the ring's warps within the warps the GPU holds.
inline cudaError_t plan_lf_step(const Geo &g, int device, const RingTable &t, StepPlan &plan) {
    int sms = 0, per_sm = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    for (int ws = 0; ws < 2; ++ws) {
        e = cudaFuncSetAttribute(step_kernel(ws != 0, t),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 step_smem(kRingSegments));
        if (e != cudaSuccess) return e;
    }
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, step_kernel(true, t),
                                                      32 * kTmaWarps, step_smem(t.nseg));
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    const int warps = sms * per_sm * kTmaWarps;
    const int S = (g.M + kFastCells - 1) / kFastCells;
    const int rows = g.L - 2;
    plan = StepPlan();
    plan.nstrips = S;
    plan.nring = (ring_count(g) + 31) / 32;
    auto bands = [&](int w) {
        const int nb = w / S;
        return nb < 1 ? 1 : (nb > rows ? rows : nb);
    };
    plan.nbands = bands(warps - plan.nring);
    if ((rows + plan.nbands - 1) / plan.nbands <= kRingAloneRows) {
        plan.alone = plan.spread = 1;
        plan.blocks = (plan.nring + S * plan.nbands + kTmaWarps - 1) / kTmaWarps;
        return cudaSuccess;
    }
    plan.spread = (long long)g.ps * 64 <= MPD_SPREAD_BYTES;
    plan.nbands = bands(warps);
    plan.nshort = (plan.nring + S - 1) / S;
    if (plan.nshort > plan.nbands) plan.nshort = plan.nbands;
    int tasks = S * plan.nbands;
    if (tasks < plan.nring) tasks = plan.nring;
    plan.blocks = (tasks + kTmaWarps - 1) / kTmaWarps;
    return cudaSuccess;
}

inline cudaError_t launch_lf_step(const Geo &g, const StepPlan &plan, const CUtensorMap &map0,
                                  const CUtensorMap &map1, double *buf0, double *buf1,
                                  DevState *st, double dt, int use_state_dt, bool want_ws,
                                  const RingTable &t, int slot, int parity,
                                  cudaStream_t stream) {
    return launch_pdl(step_kernel(want_ws, t), dim3(plan.blocks), dim3(32 * kTmaWarps),
                      step_smem(t.nseg), stream, g, map0, map1, buf0, buf1, st, dt, use_state_dt,
                      t, plan, slot, parity);
}

inline cudaError_t launch_finish_steps(const Geo &g, DevState *st, bool want_ws, int slot,
                                       cudaStream_t stream) {
    auto kernel = want_ws ? finish_steps_kernel<true> : finish_steps_kernel<false>;
    return launch_pdl(kernel, dim3(1), dim3(32), 0, stream, g, st, slot);
}

}  // namespace mpd
