// Time-stepping engine of the PyHeartSim B200 path.
//
// One persistent kernel advances every active simulation instance.  Each
// instance is owned by a "team" of CTAs that synchronise with their own bounded
// barrier, so instances of different sizes progress independently inside one
// launch.  Per step and instance:
//
//   RHS phase   RK4 reaction (simulation/simulation_gpu.py:27-43, 71-130) of
//               every voxel, then, after a team barrier, the Crank-Nicolson
//               right-hand side b = u* + dt/2 L u*  (simulation/simulation_gpu.py:245)
//               and the initial residual r0 = b - A x0  (A = I - dt/2 L, :321-322)
//   GMRES       restarted GMRES on A (CuPy semantics of the reference's call at
//               simulation/simulation_gpu.py:253): one pass and one barrier per
//               column in a Chebyshev basis, or Arnoldi with classical
//               Gram-Schmidt for stiff steps; FP64 dot products and norms
//               whatever the storage type
//   update      x += V y, then either the true-residual test of the next cycle
//               (full_cycles = 1, CuPy semantics) or the residual estimate
//               (full_cycles = 0, early exit)
//
// The Laplacian is applied matrix-free from a compacted table of six neighbour
// indices and six premultiplied coefficients per voxel, which is the CSR matrix
// of simulation/simulation_gpu.py:138-225 without the explicit zeros.
//
// Reductions are deterministic: every group of consecutive tiles of
// kThreads*VPT voxels has its own FP64 partials, and every CTA of the team sums
// the groups after the barrier in an order of their number alone.  The result
// therefore does not depend on the team size, so an instance gives
// bit-identical results alone and in a batch.
#include <cuda_runtime.h>
#include <cuda/atomic>
#include <climits>
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <algorithm>
#include <vector>
#include <map>

#include "../../include/phs.h"
#include "phs_common.cuh"

namespace phs {

// ------------------------------------------------------------------ device types
struct alignas(128) TeamSync {
    unsigned int count;    // arrivals since the launch began
    unsigned int exits;    // CTAs that have left
    unsigned int pad[30];
};

enum Action : int {
    ACT_ZERO_B = 1,      // ||b|| == 0: the solve returns b
    ACT_DONE = 2,        // residual test passed: the solve returns x
    ACT_CYCLE = 3,       // start an Arnoldi cycle (V0 holds r, s[0] = 1/||r||)
    ACT_NEXT_J = 4,      // continue the cycle with column j+1
    ACT_UPDATE_FINAL = 5,// x += V y, solve finished (Givens estimate)
    ACT_UPDATE_CHECK = 6,// x += V y, then the true-residual test
    ACT_FAIL = 7,        // non-finite norm: instance retired with an error
};

// Phase timer slots (nanoseconds of globaltimer, summed over steps).
enum ProfSlot : int {
    PF_RHS = 0, PF_RHS_WAIT, PF_A, PF_A_WAIT, PF_C, PF_C_WAIT, PF_X, PF_CHECK, PF_CHECK_WAIT,
    PF_COPY, PF_RHS1, PF_STEPS, PF_SOLVE_ITERS, PF_TEAM,
    PF_LEADER,      // time between a barrier's end and its decision: sums of the partials, solver scalars
    PF_BARRIERS,    // team barriers passed
    kProfSlots = 16
};

struct InstState {
    long long step;        // steps completed
    int id_save;           // next history slot
    int pending;           // history slot owed for the last completed step (-1: none)
    int status;
    int hbuf;              // current gate buffer
    long long arnoldi;
    long long solves;
    int max_arnoldi;
    int nonconv;
    long long arnoldi_sq;  // sum over solves of (Arnoldi steps)^2
};

template <typename T>
struct InstDev {
    const int32_t* nb;      // [n*6]
    const int16_t* nbr;     // [ldv*4] compact neighbour table (decode_nb), or nullptr
    const int32_t* nbase;   // [ldv/512*4] its base offsets per 512-voxel block
    const T* coef;          // [n*6], or nullptr when every row is isotropic (cw, m6)
    const T* cw;            // [n] common coefficient of row n (isotropic rows)
    const uint8_t* m6;      // [n] neighbour presence bits of row n (isotropic rows)
    const int32_t* enb;     // [n*12] edge pairs (a0,b0,...,a5,b5) of anisotropic rows, or nullptr
    const T* ecf;           // [n*6] edge pair coefficients, or nullptr (D0 = I)
    const uint8_t* vflags;  // [n]
    const T* vparams;       // [n*5] or nullptr
    const uint8_t* stim;    // [n_steps]
    T* u;
    T* h0;
    T* h1;
    T* x;
    T* b;
    T* V;                   // [(m+1)*n]
    T* ud;                  // [ldv*2] pairs (u*, last diffusion increment; 0 without the extrapolated guess)
    T* hist_u;              // [S*n]
    T* hist_h;              // [S*n] or nullptr
    int32_t* lat;           // [n]
    double* part;           // two buffers of part_half partial sums, [group][slot]
    TeamSync* sync;
    InstState* st;
    unsigned long long* prof;  // [kProfSlots] phase timers (CTA rank 0 of the team), or nullptr
    T params[5];
    T dt, half_dt, jmag;
    double tol, atol;
    // Chebyshev basis: interval centre and half width, T_1(-theta / delta), and
    // K_1 = (A - theta) K_0 / delta = cheb_a K_0 + cheb_b L K_0
    double theta, delta, inv_delta, t1;
    T cheb_a, cheb_b;
    long long n;
    long long ldv;          // padded voxel count (multiple of kPadVoxels): stride of V, length of per-voxel arrays
    long long n_steps;
    long long tb_steps;
    long long part_half;
    int n_tiles;
    int gt;                 // consecutive tiles of a group (the unit of the partial sums and of the CTAs' work)
    int n_groups;           // ceil(n_tiles / gt)
    int cheb;               // solves use the Chebyshev basis (cheb_rule), else Arnoldi
    int guess;
    int model;
    int m;                  // restart length actually used: min(restart, n)
    int maxiter;
    int full_cycles;
    int stride;
    int n_samples;
    int save_h;
};

// ------------------------------------------------------------------ reaction
// Mitchell-Schaeffer / Aliev-Panfilov right-hand sides,
// simulation/simulation_gpu.py:27-43 (P_2d columns 15..19 in p[0..4]).
template <typename T>
__device__ __forceinline__ void reaction(int model, T u, T h, T J, const T* p, T& du, T& dh) {
    if (model == 0) {
        du = (h * (u * u) * (T(1) - u)) / p[2] - u / p[3] + J;
        dh = (u < p[4]) ? (T(1) - h) / p[0] : -h / p[1];
    } else {
        du = -p[0] * u * (u - p[1]) * (u - T(1)) - u * h + J;
        dh = (p[2] + p[3] * h / (u + p[4])) * (-h - p[0] * u * (u - p[1] - T(1)));
    }
}

// FP32 form of the same right-hand sides: the Mitchell-Schaeffer time
// constants enter as precomputed reciprocals (q[0] = 1/tau_open, q[1] =
// 1/tau_close, q[2] = 1/tau_in, q[3] = 1/tau_out, q[4] = v_gate) and the
// Aliev-Panfilov quotient uses the fast division; FP64 keeps the reference's
// divisions exactly.
__device__ __forceinline__ void reaction_fast(int model, float u, float h, float J, const float* q, float& du,
                                              float& dh) {
    if (model == 0) {
        du = h * (u * u) * (1.0f - u) * q[2] - u * q[3] + J;
        dh = (u < q[4]) ? (1.0f - h) * q[0] : -h * q[1];
    } else {
        du = -q[0] * u * (u - q[1]) * (u - 1.0f) - u * h + J;
        dh = (q[2] + q[3] * __fdividef(h, u + q[4])) * (-h - q[0] * u * (u - q[1] - 1.0f));
    }
}

template <typename T>
__device__ __forceinline__ void reaction_any(int model, T u, T h, T J, const T* p, T& du, T& dh) {
    if constexpr (sizeof(T) == 4) reaction_fast(model, u, h, J, p, du, dh);
    else reaction(model, u, h, J, p, du, dh);
}

// Classical RK4 with J held over the step, simulation/simulation_gpu.py:71-130.
// `p` holds P_2d columns 15..19 (FP64) or their FP32 form (see reaction_fast).
template <typename T>
__device__ __forceinline__ void rk4(int model, T u, T h, T J, const T* p, T dt, T& us, T& hs) {
    T k1u, k1h, k2u, k2h, k3u, k3h, k4u, k4h;
    reaction_any(model, u, h, J, p, k1u, k1h);
    T ut = u + T(0.5) * dt * k1u;
    T ht = h + T(0.5) * dt * k1h;
    reaction_any(model, ut, ht, J, p, k2u, k2h);
    ut = u + T(0.5) * dt * k2u;
    ht = h + T(0.5) * dt * k2h;
    reaction_any(model, ut, ht, J, p, k3u, k3h);
    ut = u + dt * k3u;
    ht = h + dt * k3h;
    reaction_any(model, ut, ht, J, p, k4u, k4h);
    us = u + (dt / T(6)) * (k1u + T(2) * k2u + T(2) * k3u + k4u);
    hs = h + (dt / T(6)) * (k1h + T(2) * k2h + T(2) * k3h + k4h);
}

// P_2d columns 15..19 -> the parameter form rk4<T> expects.
template <typename T>
__host__ __device__ __forceinline__ void model_form(int model, const T* p, T* q) {
    if (sizeof(T) == 4 && model == 0) {
        q[0] = T(1) / p[0];
        q[1] = T(1) / p[1];
        q[2] = T(1) / p[2];
        q[3] = T(1) / p[3];
        q[4] = p[4];
    } else {
        for (int i = 0; i < 5; ++i) q[i] = p[i];
    }
}

// ------------------------------------------------------------------ helpers
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bound of every device-side wait: 4 s of wall time or 2^26 polls.
constexpr unsigned long long kWaitNs = 4000000000ull;
constexpr unsigned int kWaitPolls = 1u << 26;

// Bulk L2 prefetch of [p, p + bytes) (p 16-byte aligned, bytes a multiple of 16).
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned int bytes) {
    const unsigned long long g = (unsigned long long)__cvta_generic_to_global(p);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(g), "r"(bytes) : "memory");
}

// ------------------------------------------------------------------ staging ring
// Staged step kernels (RING > 0) add one producer warp to the 256 consumer
// threads.  For the update pass the consumers publish a job (the arrays the pass
// streams and their bytes per voxel); the producer copies each of the CTA's
// tiles' contiguous slices of every array into a stage of a shared-memory ring
// with 1-D cp.async.bulk, signalled on the stage's "full" mbarrier, and refills
// a stage once all consumer warps have arrived on its "empty" mbarrier.
// Consumers read the tile from shared memory; the passes that gather neighbours
// and the scattered accesses stay on global memory.
constexpr int kStageMaxArr = 12;    // arrays per stage
constexpr int kMaxStages = 6;       // ring depth limit
constexpr int kRingHeader = 1024;   // barriers and jobs ahead of the ring in dynamic shared memory

struct StageJob {
    const char* src[kStageMaxArr];  // array base (voxel 0)
    int bytes[kStageMaxArr];        // bytes of one tile's slice
    int off[kStageMaxArr];          // offset of the slice in a stage
    int n_arr;
    int stage_bytes;
    int n_stages;
    int tile0, step, gt, n_tiles;   // the CTA's groups of gt tiles: tile0, tile0 + step, ...; tiles < n_tiles
    int quit;
};
struct RingHeader {
    unsigned long long full[kMaxStages];
    unsigned long long empty[kMaxStages];
    StageJob job[2];
    int stop;                       // a bounded stage wait gave up: later waits return at once
};
static_assert(sizeof(RingHeader) <= kRingHeader, "ring header");

// Consumer-only CTA barrier: __syncthreads without a producer warp, else named
// barrier 1 over the 256 consumer threads.
template <bool ST>
__device__ __forceinline__ void csync() {
    if constexpr (ST) asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
    else __syncthreads();
}
// Job hand-over on named barrier 2: consumers arrive, the producer waits.
__device__ __forceinline__ void job_arrive() { asm volatile("bar.arrive 2, %0;" ::"n"(kThreads + 32) : "memory"); }
__device__ __forceinline__ void job_wait() { asm volatile("bar.sync 2, %0;" ::"n"(kThreads + 32) : "memory"); }

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t a, unsigned int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t a) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t a, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    return ok != 0u;
}
// Bounded wait for the phase of parity `parity` of the mbarrier at a.  Gives up
// after 4 s or 2^26 polls (sets *stop and the abort word), and at once once
// *stop is set when `heed_stop`; returns whether the phase completed.
__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity, volatile int* stop, unsigned int* abort_word,
                                          bool heed_stop = true) {
    if (mbar_try(a, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (unsigned int polls = 0;; ++polls) {
        if (mbar_try(a, parity)) return true;
        if (heed_stop && *stop) return false;
        if (polls > kWaitPolls || global_ns() - t0 > kWaitNs) {
            *stop = 1;
            atomicOr(abort_word, 1u);
            return false;
        }
    }
}
// 1-D bulk copy global -> shared (both 16-byte aligned, bytes a multiple of 16),
// completion counted on the mbarrier at mbar.  No multicast.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"((unsigned long long)__cvta_generic_to_global(src)), "r"(bytes), "r"(mbar)
                 : "memory");
}
// Orders this thread's generic-proxy global accesses before later async-proxy
// (bulk copy) ones.
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// Consumer side of the staging ring.  A phase lists its arrays with add()
// (every consumer thread makes the same calls, so all agree on the offsets;
// thread 0 writes the job), then publish() hands the job to the producer and
// returns the ring depth, 0 when the phase runs unstaged; acquire() waits for
// the next tile's stage and release() marks the calling warp done with it.
template <int RING, int TILE, typename T>
struct Stager {
    RingHeader* rh;
    unsigned char* ring;
    int job_buf;
    int lay_off, lay_n;
    int nst, sg;          // ring depth of the phase, stage of the current tile
    unsigned int cpar;    // parity to wait for on each full barrier

    __device__ __forceinline__ void begin() {
        lay_off = 0;
        lay_n = 0;
    }
    __device__ __forceinline__ int add(const void* base, int elem) {
        const int o = lay_off;
        if (threadIdx.x == 0 && lay_n < kStageMaxArr) {
            StageJob& J = rh->job[job_buf];
            J.src[lay_n] = static_cast<const char*>(base);
            J.bytes[lay_n] = TILE * elem;
            J.off[lay_n] = o;
        }
        lay_off += TILE * elem;
        ++lay_n;
        return o;
    }
    // basis vectors a phase may stage after its fixed arrays: as many as keep
    // the ring at least two stages deep
    __device__ __forceinline__ int vec_cap() const {
        const int c = (RING / 2 - lay_off) / (TILE * (int)sizeof(T));
        return max(0, min(c, kStageMaxArr - lay_n));
    }
    __device__ __forceinline__ int publish(int rank, int P, int n_tiles, int n_groups, int gt) {
        nst = (lay_off > 0 && lay_n <= kStageMaxArr) ? RING / lay_off : 0;
        if (nst > kMaxStages) nst = kMaxStages;
        if (rank >= n_groups) nst = 0;
        if (nst == 0) return 0;
        if (threadIdx.x == 0) {
            StageJob& J = rh->job[job_buf];
            J.n_arr = lay_n;
            J.stage_bytes = lay_off;
            J.n_stages = nst;
            J.tile0 = rank;
            J.step = P;
            J.gt = gt;
            J.n_tiles = n_tiles;
            J.quit = 0;
        }
        fence_proxy_async_global();   // this thread's global writes before the bulk reads
        csync<true>();
        job_arrive();
        job_buf ^= 1;
        sg = -1;
        return nst;
    }
    __device__ __forceinline__ const unsigned char* acquire(unsigned int* abort_word) {
        if (++sg == nst) sg = 0;
        mbar_wait(smem_u32(&rh->full[sg]), (cpar >> sg) & 1u, &rh->stop, abort_word);
        cpar ^= 1u << sg;
        return ring + sg * lay_off;
    }
    __device__ __forceinline__ void release() {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(smem_u32(&rh->empty[sg]));
    }
    // hands the producer warp its last job
    __device__ __forceinline__ void quit() {
        if (threadIdx.x == 0) rh->job[job_buf].quit = 1;
        csync<true>();
        job_arrive();
    }
};

struct SharedCtl {
    int abort;
    int action;
    int k;            // basis vectors of the update that follows
    int settled;      // the cycle's estimate is below rounding level (kSettled)
    double bnorm, atol_eff;
    double rnorm;     // residual at the start of the cycle
    int cheb;         // form of the solve's cycles from here on: Chebyshev basis, else Arnoldi
    int iters_cap;    // columns of the solve as maxiter counts them
    int iters_short;  // columns of the early exit's short cycles, which it does not
    int refined;      // the columns after a settled full cycle have run
    double sj;        // Arnoldi: scale of the column the next pass applies A to
    double sz;        // Chebyshev basis: sum of z_i^2
};

// Bounded team barrier: every CTA of the team arrives on one counter and polls
// it until the team's `target` is reached.  No CTA leads: what a barrier
// combines (partial sums, solver scalars) every CTA computes for itself from
// the partials, in the same order and so to the same bits.  That takes three
// dependent L2 round trips out of a barrier (the leader's read of the partials,
// its release and the waiters' read of its results): 5.3-7.5 us with a leader
// that reduced, 3.8-4.3 us now with sums and decision (7 to 157 CTAs).
//
// Ordering: the arrival is a release RMW after a CTA barrier (cumulative over
// the CTA's writes), the poll an acquire load, followed by a CTA barrier.
// Returns false when the wait gave up or another team aborted; the kernel then
// leaves all loops.  A team of one CTA needs its own CTA barrier only.
template <bool ST>
__device__ __forceinline__ bool team_barrier(TeamSync* ts, int P, unsigned int target, unsigned int* abort_word,
                                             SharedCtl& ctl) {
    csync<ST>();
    if (P == 1) return true;
    if (threadIdx.x == 0) {
        cuda::atomic_ref<unsigned int, cuda::thread_scope_device> cnt(ts->count);
        cnt.fetch_add(1u, cuda::memory_order_release);
        unsigned long long t0 = 0;
        for (unsigned int polls = 0; (int)(cnt.load(cuda::memory_order_acquire) - target) < 0; ++polls) {
            if ((polls & 63u) != 63u) continue;
            cuda::atomic_ref<unsigned int, cuda::thread_scope_device> ab(*abort_word);
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            if (ab.load(cuda::memory_order_relaxed) != 0u) { ctl.abort = 1; break; }
            if (polls > kWaitPolls || now - t0 > kWaitNs) {
                ab.fetch_or(1u, cuda::memory_order_relaxed);
                ctl.abort = 1;
                break;
            }
        }
    }
    csync<ST>();
    return ctl.abort == 0;
}

// The six (neighbour, coefficient) pairs of row n, as 8/16-byte vector loads.
__device__ __forceinline__ void load_nb(const int32_t* nb, long long n, int32_t (&q)[6]) {
    const int2* p = reinterpret_cast<const int2*>(nb + 6 * n);
    int2 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
    q[0] = a.x; q[1] = a.y; q[2] = b.x; q[3] = b.y; q[4] = c.x; q[5] = c.y;
}
__device__ __forceinline__ void load_coef(const float* cf, long long n, float (&c)[6]) {
    const float2* p = reinterpret_cast<const float2*>(cf + 6 * n);
    float2 a = __ldg(p), b = __ldg(p + 1), d = __ldg(p + 2);
    c[0] = a.x; c[1] = a.y; c[2] = b.x; c[3] = b.y; c[4] = d.x; c[5] = d.y;
}
__device__ __forceinline__ void load_coef(const double* cf, long long n, double (&c)[6]) {
    const double2* p = reinterpret_cast<const double2*>(cf + 6 * n);
    double2 a = __ldg(p), b = __ldg(p + 1), d = __ldg(p + 2);
    c[0] = a.x; c[1] = a.y; c[2] = b.x; c[3] = b.y; c[4] = d.x; c[5] = d.y;
}

// Compact neighbour table.  In the row order of a lattice (x fastest) the
// present +x and -x neighbours of voxel n are n + 1 and n - 1 (slots 0 and 1
// of the reference's column order), and the other four slots hold offsets that
// change slowly along the rows: base[r] of the voxel's 512-voxel block plus the
// voxel's int16 residual r (slots 2..5).  Exact for every present neighbour
// (checked when the table is built); absent ones decode to unused values.
__device__ __forceinline__ void decode_nb(short4 r, int4 b, long long n, int32_t (&q)[6]) {
    const int32_t nn = (int32_t)n;
    q[0] = nn + 1;
    q[1] = nn - 1;
    q[2] = nn + b.x + r.x;
    q[3] = nn + b.y + r.y;
    q[4] = nn + b.z + r.z;
    q[5] = nn + b.w + r.w;
}

// One value, or the pair (u*, last diffusion increment), per voxel.
template <typename T>
struct Pair;
template <>
struct Pair<float> { using type = float2; };
template <>
struct Pair<double> { using type = double2; };
template <typename T>
using PairT = typename Pair<T>::type;

__device__ __forceinline__ float lap_zero(float) { return 0.f; }
__device__ __forceinline__ double lap_zero(double) { return 0.0; }
__device__ __forceinline__ float2 lap_zero(float2) { return make_float2(0.f, 0.f); }
__device__ __forceinline__ double2 lap_zero(double2) { return make_double2(0.0, 0.0); }
// s += g - o
__device__ __forceinline__ void add_diff(float& s, float g, float o) { s += g - o; }
__device__ __forceinline__ void add_diff(double& s, double g, double o) { s += g - o; }
__device__ __forceinline__ void add_diff(float2& s, float2 g, float2 o) { s.x += g.x - o.x; s.y += g.y - o.y; }
__device__ __forceinline__ void add_diff(double2& s, double2 g, double2 o) { s.x += g.x - o.x; s.y += g.y - o.y; }
// s += c * (g - o)
template <typename T>
__device__ __forceinline__ void add_scaled(T& s, T c, T g, T o) { s += c * (g - o); }
__device__ __forceinline__ void add_scaled(float2& s, float c, float2 g, float2 o) {
    s.x += c * (g.x - o.x);
    s.y += c * (g.y - o.y);
}
__device__ __forceinline__ void add_scaled(double2& s, double c, double2 g, double2 o) {
    s.x += c * (g.x - o.x);
    s.y += c * (g.y - o.y);
}
template <typename T>
__device__ __forceinline__ T times(T c, T s) { return c * s; }
__device__ __forceinline__ float2 times(float c, float2 s) { return make_float2(c * s.x, c * s.y); }
__device__ __forceinline__ double2 times(double c, double2 s) { return make_double2(c * s.x, c * s.y); }

// Matrix-free rows of L applied to `vec` at the thread's voxels n0 + v * kThreads
// of a tile (own[v] = vec there).  Nothing is stored in between, so the loads
// of all VPT voxels (tables, then gathers) are in flight together: with a store
// after each voxel, as this was written before, every voxel waited for its own
// table and gathers in turn.  No bounds test: the per-voxel arrays are padded
// to whole tiles with zeros, and a row of zero coefficients reads itself.
// Isotropic rows (D0 = I: one coefficient c_n / Delta^2 on every present
// neighbour) sum the differences first; other rows have six coefficients, and
// the edge cross terms of simulation/simulation_gpu.py:199-217 as six
// antisymmetric pairs.  NB: 0 int32 table, 1 compact table, 2 the instance's.
template <typename T, int VPT, bool EDGE, int NB, typename V>
__device__ __forceinline__ void tile_lap(const InstDev<T>& I, const V* vec, long long n0, bool tb, const V (&own)[VPT],
                                         V (&lap)[VPT]) {
    const bool compact = NB == 1 || (NB == 2 && I.nbr != nullptr);
    if (I.cw) {
        unsigned mk[VPT];
        T w[VPT];
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            const long long n = n0 + v * kThreads;
            mk[v] = __ldg(I.m6 + n);
            w[v] = __ldg(I.cw + n);
            // a zero coefficient reads nothing: its stored offset may be anything
            if (w[v] == T(0) || (tb && (__ldg(I.vflags + n) & PHS_VFLAG_TBLOCK))) mk[v] = 0u;
        }
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            const long long n = n0 + v * kThreads;
            int32_t q[6];
            if (compact)
                decode_nb(__ldg(reinterpret_cast<const short4*>(I.nbr) + n),
                          __ldg(reinterpret_cast<const int4*>(I.nbase) + (n >> 9)), n, q);
            else
                load_nb(I.nb, n, q);
            V g[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) g[k] = vec[((mk[v] >> k) & 1u) ? q[k] : (int32_t)n];
            V s = lap_zero(own[v]);
#pragma unroll
            for (int k = 0; k < 6; ++k) add_diff(s, g[k], own[v]);
            lap[v] = times(w[v], s);
        }
    } else {
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            const long long n = n0 + v * kThreads;
            int32_t q[6];
            T c[6];
            if (compact)
                decode_nb(__ldg(reinterpret_cast<const short4*>(I.nbr) + n),
                          __ldg(reinterpret_cast<const int4*>(I.nbase) + (n >> 9)), n, q);
            else
                load_nb(I.nb, n, q);
            load_coef(I.coef, n, c);
            V g[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) g[k] = vec[c[k] != T(0) ? q[k] : (int32_t)n];
            V s = lap_zero(own[v]);
#pragma unroll
            for (int k = 0; k < 6; ++k) add_scaled(s, c[k], g[k], own[v]);
            if (EDGE && I.ecf) {
                const int4* pi = reinterpret_cast<const int4*>(I.enb + 12 * n);
                const int4 i0 = __ldg(pi), i1 = __ldg(pi + 1), i2 = __ldg(pi + 2);
                const int32_t e[12] = {i0.x, i0.y, i0.z, i0.w, i1.x, i1.y, i1.z, i1.w, i2.x, i2.y, i2.z, i2.w};
                load_coef(I.ecf, n, c);
                V a[6], b[6];
#pragma unroll
                for (int p = 0; p < 6; ++p) {
                    a[p] = vec[c[p] != T(0) ? e[2 * p] : (int32_t)n];
                    b[p] = vec[c[p] != T(0) ? e[2 * p + 1] : (int32_t)n];
                }
#pragma unroll
                for (int p = 0; p < 6; ++p) add_scaled(s, c[p], a[p], b[p]);
            }
            if (tb && (__ldg(I.vflags + n) & PHS_VFLAG_TBLOCK)) s = lap_zero(own[v]);
            lap[v] = s;
        }
    }
}

// Sums of N values over a warp, N a power of two: the halves of the value list
// go to the halves of the warp at each exchange, so N sums take N - 1 + 5 -
// log2(N) exchanges instead of 5 N.  Lane l returns the sum of value
// l >> (5 - log2(N)); the order of the additions is fixed.
template <int N>
__device__ __forceinline__ double warp_sums(double (&v)[N], int lane) {
    int off = 16;
#pragma unroll
    for (int h = N / 2; h >= 1; h /= 2) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double send = up ? v[i] : v[i + h];
            const double keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
        off /= 2;
    }
    for (; off >= 1; off /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    return v[0];
}
__host__ __device__ constexpr int log2_of(int n) { return n <= 1 ? 0 : 1 + log2_of(n / 2); }

// Basis vectors whose loads and sums are taken together: FP32 tiles hold two or
// four voxels per thread (as many loads per vector), FP64 tiles one, and the FP64
// plain form passes over some twenty vectors per column (160k voxels, 30 steps:
// 9.9 ms by eights, 10.7 by sixteens with their spills, 10.2 by fours).
template <typename T>
constexpr int kChunkOf = sizeof(T) == 8 ? 8 : 4;
// A full GMRES cycle ends early once its residual estimate is at most this
// fraction of ||b||: half a unit roundoff of the stored type.  With isotropic rows
// A is I - dt/2 L with eigenvalues of 1 and above, so what the remaining columns
// could add to x is below a rounding of x (anisotropic rows: unproven, but ||A^-1||
// is near 1 there too, and the true-residual test follows either way); besides,
// classical Gram-Schmidt has lost the basis'
// orthogonality by then (|v_0 . v_j| of 0.1 to 1 where the estimate passes this
// line) and those columns are rounding noise.  On the sheet and shell runs the
// line is crossed after 18-26 of 50 columns with the error against the exact
// solution unchanged (2.5e-16 relative at column 21 and at column 50); at
// larger steps (dt/2 max(-L_nn) above ~5) it is not reached and the cycle runs
// to its end.
template <typename T>
constexpr double kSettled = sizeof(T) == 8 ? 5.5511151231257827e-17 : 2.9802322387695312e-08;

// A full cycle in the Chebyshev basis whose true residual is above this fraction
// of ||b|| (rounding level of the residual itself is 1-2e-16 ||b||) is followed by
// a few columns more: where r0 is near ||b|| (the edges of a fresh stimulus) the
// roundings of the three-term recurrence, which scale with r0, are above those
// of b (1.4e-15 ||b|| at r0 = 0.3 ||b||, 2e-16 after).
template <typename T>
constexpr double kRefine = sizeof(T) == 8 ? 4.4408920985006262e-16 : 2.384185791015625e-07;

// Partial sums are kept per group of consecutive tiles (one tile, more for
// instances of more than this many tiles), whatever CTA a group falls to, so
// that no team has to read many of them: every CTA sums all groups.
constexpr int kMaxGroupsF32 = 640, kMaxGroupsF64 = 444;
constexpr int kSumLoads = 8;                  // partials a thread loads together
constexpr int kRedDoubles = 16 * kSlots;      // warp sums a CTA holds back before it combines them
constexpr int kTri = (kMaxRestart + 1) * (kMaxRestart + 2) / 2;
__device__ __forceinline__ int tri(int row) { return row * (row + 1) / 2; }

// A solve whose squared residual norm is below this (||r|| < 1e-50: resting tissue
// long after its last wave, solved to a tolerance without an absolute part) is
// Arnoldi's, whose vectors are normalised: the Chebyshev form sums squares of
// 1 / ||r||, which leave the range of FP64 as the estimate passes 1e-154.
constexpr double kTinySquare = 1e-100;

// Below this share of <K_j, K_j> the part of K_j outside the span of the
// earlier vectors is zero (breakdown) or lost to rounding.
constexpr double kPivot = 1e-12;

// ------------------------------------------------------------------ the kernel
// Each solve (I - dt/2 L) x = b is restarted GMRES, in one of two forms:
//
//  Chebyshev basis (I.cheb, the rule is cheb_rule's): the Krylov vectors are
//  K_j = T_j((A - theta) / delta) r0 for the interval [theta - delta, theta +
//  delta] that Gershgorin's theorem gives for A (isotropic rows; a heuristic for
//  anisotropic ones, see make_dev), a basis well enough conditioned to be used
//  without orthogonalising it.  Column j is ONE pass over the voxels
//  (K_{j+1} from K_j and K_{j-1}, and its dots with every K_i) and ONE team
//  barrier.  From the Gram matrix G of the dots (FP64) every CTA keeps
//  W = R^-T, G = R^T R, and z = W t, t_i = T_i(-theta / delta): with the
//  residuals written as sum c_i K_i under sum c_i t_i = 1 (a polynomial that is
//  1 at 0), the GMRES residual is 1 / ||z|| and its coefficients W^T z /
//  ||z||^2.  The iterates, estimates and column counts are those of Arnoldi
//  GMRES (FP32: solutions agree to 1e-8, estimates to 3 digits at tol 1e-7;
//  FP64: to 1e-15), which needed two passes and two barriers per column, the
//  second pass to orthogonalise.  200 x 200 sheet: FP32 70 -> 24 us per step of
//  3 columns, FP64 460 -> 157 us per step of 22.
//
//  Arnoldi with classical Gram-Schmidt (the others: stiff steps with long
//  cycles): phase A applies A and takes the dots, phase C orthogonalises.
//
// EDGE: the launch carries anisotropic instances (edge cross terms); the
// isotropic launches compile without that code.  RING > 0: a producer warp
// copies the update pass's slices into a shared-memory ring.
template <typename T, int VPT, int MINB, bool EDGE, int RING, bool NBC>
__global__ void __launch_bounds__(kThreads + (RING > 0 ? 32 : 0), MINB)
step_kernel(const InstDev<T>* __restrict__ insts, const int4* __restrict__ cta_map,
            long long n_steps_launch, unsigned int* abort_word) {
    constexpr bool ST = RING > 0;   // staged: producer warp + shared-memory ring (FP32 only)
    static_assert(!ST || sizeof(T) == 4, "staged kernels are FP32");
    // NBC: every instance of the launch has a compact neighbour table (decode_nb)
    static_assert(!(ST && NBC), "staged kernels choose the table per instance");
    constexpr int NB = ST ? 2 : (NBC ? 1 : 0);
    constexpr int TILE = kThreads * VPT;
    constexpr int kChunk = kChunkOf<T>;
    using P2 = PairT<T>;
    const int4 cm = cta_map[blockIdx.x];
    const int rank = cm.y;
    const int P = cm.z;
    const bool pf_on = cm.w != 0;

    __shared__ InstDev<T> I;
    __shared__ SharedCtl ctl;
    __shared__ long long sh_step0;
    __shared__ int sh_id_save, sh_pending, sh_hbuf, sh_status;
    // solver scalars: R^-T of the Gram matrix or R of the Hessenberg QR (both
    // triangular), vectors over the columns
    __shared__ double tm[kTri];
    __shared__ double va[kMaxRestart + 2], vb[kMaxRestart + 2], vc[kMaxRestart + 2], vd[kMaxRestart + 2];
    __shared__ double gsum[kSlots];                 // sums of the barrier that just ended
    __shared__ double shc[kMaxRestart + 1];         // coefficients of the next pass
    __shared__ double red[kRedDoubles];
    __shared__ double bs[kThreads];
    // staged kernels: ring header (mbarriers, jobs) and the ring itself
    extern __shared__ __align__(128) unsigned char dyn_smem[];
    RingHeader* const rh = reinterpret_cast<RingHeader*>(dyn_smem);
    unsigned char* const ring = dyn_smem + kRingHeader;

    if (threadIdx.x == 0) {
        I = insts[cm.x];
        sh_step0 = __ldcg(&I.st->step);
        sh_id_save = __ldcg(&I.st->id_save);
        sh_pending = __ldcg(&I.st->pending);
        sh_hbuf = __ldcg(&I.st->hbuf);
        sh_status = __ldcg(&I.st->status);
        ctl.abort = 0;
        if constexpr (ST) {
            for (int q = 0; q < kMaxStages; ++q) {
                mbar_init(smem_u32(&rh->full[q]), 1u);
                mbar_init(smem_u32(&rh->empty[q]), (unsigned)kWarps);
            }
            rh->stop = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    __syncthreads();

    if constexpr (ST) {
        // ---- producer warp: copies the slices of each published job's tiles
        if (threadIdx.x >= kThreads) {
            const int pl = threadIdx.x - kThreads;
            const uint32_t ring_u32 = smem_u32(ring);
            volatile int* stop = &rh->stop;
            unsigned int epar = 0xffffffffu;   // parity to wait for on each empty barrier (fresh: passes)
            unsigned int fpar = 0u;            // fills of each stage, mod 2
            unsigned int used = 0u;
            bool dead = false;                 // an empty-barrier wait gave up: issue nothing more
            int jb = 0;
            for (;;) {
                job_wait();
                const StageJob* J = &rh->job[jb];
                jb ^= 1;
                if (J->quit) break;
                fence_proxy_async_global();
                const int na = J->n_arr, sbytes = J->stage_bytes, nst = J->n_stages;
                const int tstep = J->step, nt = J->n_tiles, gt = J->gt;
                const char* src = pl < na ? J->src[pl] : nullptr;
                const int bytes = pl < na ? J->bytes[pl] : 0;
                const int off = pl < na ? J->off[pl] : 0;
                int sg = 0;
                for (int grp = J->tile0; grp * gt < nt && !dead; grp += tstep) {
                    const int tend = min(nt, (grp + 1) * gt);
                    for (int tile = grp * gt; tile < tend && !dead; ++tile) {
                        const uint32_t fb = smem_u32(&rh->full[sg]);
                        bool ok = true;
                        if (pl == 0) ok = mbar_wait(smem_u32(&rh->empty[sg]), (epar >> sg) & 1u, stop, abort_word);
                        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                        if (!ok) {
                            dead = true;
                            break;
                        }
                        epar ^= 1u << sg;
                        if (pl == 0) mbar_expect_tx(fb, (uint32_t)sbytes);
                        __syncwarp();
                        if (pl < na)
                            bulk_g2s(ring_u32 + (uint32_t)(sg * sbytes + off), src + (size_t)tile * bytes,
                                     (uint32_t)bytes, fb);
                        fpar ^= 1u << sg;
                        used |= 1u << sg;
                        if (++sg == nst) sg = 0;
                    }
                }
            }
            // every copy this CTA issued has landed before it exits
            if (pl == 0)
                for (int q = 0; q < kMaxStages; ++q)
                    if ((used >> q) & 1u) mbar_wait(smem_u32(&rh->full[q]), ((fpar >> q) & 1u) ^ 1u, stop, abort_word, false);
            __syncwarp();
            return;
        }
    }

    const long long N = I.n;
    const int gt = I.gt, n_groups = I.n_groups, n_tiles = I.n_tiles;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const bool cheb = I.cheb != 0;
    long long step = sh_step0;
    long long step_end = step + n_steps_launch;
    if (step_end > I.n_steps) step_end = I.n_steps;
    int id_save = sh_id_save;
    int pending = sh_pending;
    int hbuf = sh_hbuf;
    bool retired = (sh_status == PHS_ERR_NONFINITE);
    bool aborted = false;
    // solve statistics of this launch (thread 0 of rank 0)
    __shared__ long long st_arnoldi, st_arnoldi_sq, st_solves;
    __shared__ int st_max_arnoldi, st_nonconv;
    if (threadIdx.x == 0) {
        st_arnoldi = st_arnoldi_sq = st_solves = 0;
        st_max_arnoldi = st_nonconv = 0;
    }
    // optional phase timer: thread 0 of CTA rank 0 of each team
    __shared__ unsigned long long pf[kProfSlots];
    __shared__ unsigned long long pf_t;
    const bool prof_on = (I.prof != nullptr) && rank == 0;
    if (prof_on && threadIdx.x == 0) {
        for (int i = 0; i < kProfSlots; ++i) pf[i] = 0ull;
        pf_t = global_ns();
    }
    auto mark = [&](int slot) {
        if (prof_on && threadIdx.x == 0) {
            unsigned long long t = global_ns();
            pf[slot] += t - pf_t;
            pf_t = t;
        }
    };
    unsigned int target = 0;
    auto barrier = [&]() -> bool {
        target += (unsigned int)P;
        const bool ok = team_barrier<ST>(I.sync, P, target, abort_word, ctl);
        if (prof_on && threadIdx.x == 0) pf[PF_BARRIERS] += 1;
        return ok;
    };

    // ---- partial sums.  A warp's sum of a tile goes to red[entry][warp][slot]
    // (entry: the CTA's groups since the last flush; the tiles of a group add
    // up), flush() adds the warps in order into the group's partials in global
    // memory.  Two partial buffers alternate: a CTA may write the next phase's
    // partials while another still reads this one's.
    int pbuf = 0;
    int entries = 0, group0 = 0;
    double* const part0 = I.part;
    auto phase_begin = [&]() {
        entries = 0;
        group0 = rank;
    };
    auto flush = [&](int ns, bool more) {
        csync<ST>();
        double* dst = part0 + (size_t)pbuf * I.part_half;
        for (int e = threadIdx.x; e < entries * ns; e += kThreads) {
            const int q = e / ns, s = e - q * ns;
            double a = 0.0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) a += red[(q * kWarps + w) * ns + s];
            dst[(size_t)(group0 + q * P) * ns + s] = a;
        }
        if (more) csync<ST>();
        group0 += entries * P;
        entries = 0;
    };
    // a lane's sums of slot s for the current group
    auto put = [&](int ns, int s, double v, bool first) {
        double* p = &red[(entries * kWarps + warp) * ns + s];
        *p = first ? v : *p + v;
    };
    auto group_done = [&](int ns) {
        ++entries;
        if ((entries + 1) * kWarps * ns > kRedDoubles) flush(ns, true);
    };
    // sums over all groups into gsum[0..ns), in an order that depends on the
    // number of groups alone: thread t adds slot t % ns over every
    // (256 / ns)-th group, then a warp, or eight lanes, per slot add the threads.
    auto reduce = [&](int ns) {
        const double* src = part0 + (size_t)pbuf * I.part_half;
        const int stride = kThreads / ns;
        const int q0 = threadIdx.x / ns, s = threadIdx.x - q0 * ns;
        double a = 0.0;
        if (q0 < stride) {
            // kSumLoads loads in flight whatever the count (a remainder loop would
            // wait for each of its loads in turn)
            for (int q = q0; q < n_groups; q += kSumLoads * stride) {
                double v[kSumLoads];
#pragma unroll
                for (int i = 0; i < kSumLoads; ++i)
                    v[i] = (q + i * stride < n_groups) ? __ldcg(src + (size_t)(q + i * stride) * ns + s) : 0.0;
#pragma unroll
                for (int i = 0; i < kSumLoads; ++i) a += v[i];
            }
        }
        bs[threadIdx.x] = a;
        csync<ST>();
        const int live = min(stride, n_groups);
        if (ns <= kWarps) {              // a warp per slot
            if (warp < ns) {
                double b = 0.0;
                for (int l = lane; l < live; l += 32) b += bs[l * ns + warp];
                b = warp_sum(b);
                if (lane == 0) gsum[warp] = b;
            }
        } else {                         // eight lanes per slot
            for (int t0 = 0; t0 < ns; t0 += 4 * kWarps) {
                const int t = t0 + 4 * warp + (lane >> 3);
                double b = 0.0;
                if (t < ns)
                    for (int l = lane & 7; l < live; l += 8) b += bs[l * ns + t];
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
                if ((lane & 7) == 0 && t < ns) gsum[t] = b;
            }
        }
        csync<ST>();
        pbuf ^= 1;
    };
    // the barrier of a phase that summed ns slots
    unsigned long long t_red = 0;
    auto barrier_sums = [&](int ns) -> bool {
        flush(ns, false);
        if (!barrier()) return false;
        if (prof_on && threadIdx.x == 0) t_red = global_ns();
        reduce(ns);
        return true;
    };
    auto decided = [&]() {   // after every CTA's own decision
        csync<ST>();
        if (prof_on && threadIdx.x == 0) pf[PF_LEADER] += global_ns() - t_red;
    };
    auto voxel = [&](int tile, int v) -> long long { return (long long)tile * TILE + v * kThreads + threadIdx.x; };

    // ---- consumer side of the staging ring (ST)
    Stager<RING, TILE, T> stg{rh, ring, 0, 0, 0, 0, 0, 0u};

    // Prefetch into L2 the slice of an array (elem bytes per voxel) that `tile`
    // will read, so that the loads of the CTA's next tile find it there; one lane
    // per array, spread over the warps.  Only in launches whose working set is a
    // multiple of L2 (plan_prefetch).  Start and end are rounded down to 16
    // bytes: every prefetched byte lies inside the array (whose allocation starts
    // 256-byte aligned).
    auto pf_slice = [&](const void* arr, int elem, int tile) {
        if (arr == nullptr || tile >= n_tiles) return;
        const long long v0 = (long long)tile * TILE;
        const long long v1 = (v0 + TILE < N) ? v0 + TILE : N;
        uintptr_t a = reinterpret_cast<uintptr_t>(arr) + (uintptr_t)(v0 * elem);
        uintptr_t b = reinterpret_cast<uintptr_t>(arr) + (uintptr_t)(v1 * elem);
        a &= ~(uintptr_t)15;
        b &= ~(uintptr_t)15;
        if (b > a) prefetch_l2(reinterpret_cast<const void*>(a), (unsigned int)(b - a));
    };
    // the row tables of the operator (neighbours, coefficients, flags, edges)
    auto pf_rows = [&](int t, int tile) {
        switch (t) {
            case 0: if (NB == 1 || (NB == 2 && I.nbr)) pf_slice(I.nbr, 8, tile); else pf_slice(I.nb, 24, tile); break;
            case 1: pf_slice(I.cw ? (const void*)I.cw : (const void*)I.coef, I.cw ? (int)sizeof(T) : 6 * (int)sizeof(T), tile); break;
            case 2: pf_slice(I.m6, 1, tile); break;
            case 3: if (EDGE) pf_slice(I.enb, 48, tile); break;
            case 4: if (EDGE) pf_slice(I.ecf, 6 * (int)sizeof(T), tile); break;
            default: break;
        }
    };
    constexpr int kRowArrays = 5;
    // the CTA's tile after `tile` of group `grp`
    auto tile_after = [&](int grp, int tile) {
        return (tile + 1 < min(n_tiles, (grp + 1) * gt)) ? tile + 1 : (grp + P) * gt;
    };

    auto params_of = [&](long long n, T* p) {
        if (I.vparams) {
            T raw[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) raw[q] = I.vparams[5 * n + q];
            model_form<T>(I.model, raw, p);
        } else {
#pragma unroll
            for (int q = 0; q < 5; ++q) p[q] = I.params[q];
        }
    };

    T* const Vb = I.V;
    P2* const UD = reinterpret_cast<P2*>(I.ud);
    const size_t ldV = (size_t)I.ldv;

    // ---- what every CTA decides from the sums of a barrier ------------------
    int iters_solve = 0, cols = 0;   // columns of the solve, of the cycle
    auto fail = [&]() {
        ctl.action = ACT_FAIL;
        if (rank == 0) I.st->status = PHS_ERR_NONFINITE;
    };
    auto account_solve = [&]() {
        if (rank == 0 && threadIdx.x == 0 && iters_solve > 0) {
            st_arnoldi += iters_solve;
            st_arnoldi_sq += (long long)iters_solve * iters_solve;
            st_solves += 1;
            st_max_arnoldi = max(st_max_arnoldi, iters_solve);
        }
    };
    // start of a cycle from the residual in column 0, squared norm r2 (thread 0)
    auto start_cycle = [&](double r2) {
        ctl.action = ACT_CYCLE;
        const double w0 = rsqrt(r2);
        ctl.rnorm = r2 * w0;
        if (cheb && ctl.cheb) {
            tm[0] = w0;            // W
            va[0] = w0;            // z
            vb[0] = 1.0;           // t
            ctl.sz = w0 * w0;
        } else {
            va[0] = r2 * w0;       // g
            vb[0] = w0;            // s
            ctl.sj = vb[0];
        }
    };
    auto decide_rhs = [&]() {
        if (threadIdx.x == 0) {
            ctl.cheb = cheb && !(gsum[1] < kTinySquare);
            ctl.iters_cap = ctl.iters_short = ctl.refined = 0;
            const double bn = sqrt(gsum[0]), rn = sqrt(gsum[1]);
            const double atol_eff = fmax(I.atol, I.tol * bn);
            ctl.bnorm = bn;
            ctl.atol_eff = atol_eff;
            if (!isfinite(bn) || !isfinite(rn)) fail();
            else if (bn == 0.0) ctl.action = ACT_ZERO_B;
            else if (rn <= atol_eff) ctl.action = ACT_DONE;
            else start_cycle(gsum[1]);
        }
        decided();
    };
    // Chebyshev basis, column j (K_0..K_{j+1} there, gsum[i] = <K_{j+1}, K_i>):
    // the next row of W and entry of z, the residual estimate, and at the end of
    // a cycle the coefficients of x = x0 + sum y_i K_i.  One warp.
    auto decide_cheb = [&](int j, int cycle_cols) {
        if (warp == 0) {
            const double gjj = gsum[j + 1];
            // x = W g, the new column of R (four chains of products per lane)
            double s2[2] = {0.0, 0.0};      // x.x, x.z
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = lane + 32 * h;
                if (i <= j) {
                    const double* wr = tm + tri(i);
                    double a[4] = {0.0, 0.0, 0.0, 0.0};
                    int l = 0;
                    for (; l + 3 <= i; l += 4) {
#pragma unroll
                        for (int t = 0; t < 4; ++t) a[t] += wr[l + t] * gsum[l + t];
                    }
                    for (; l <= i; ++l) a[0] += wr[l] * gsum[l];
                    const double x = (a[0] + a[1]) + (a[2] + a[3]);
                    s2[0] += x * x;
                    s2[1] += x * va[i];
                    vd[i] = x;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                s2[0] += __shfl_xor_sync(0xffffffffu, s2[0], o);
                s2[1] += __shfl_xor_sync(0xffffffffu, s2[1], o);
            }
            __syncwarp();
            const double tj = (j == 0) ? I.t1 : 2.0 * I.t1 * vb[j] - vb[j - 1];
            double p2 = gjj - s2[0];
            const bool finite = isfinite(gjj) && isfinite(s2[0]);
            const bool dependent = fabs(p2) <= kPivot * gjj;        // breakdown: K_{j+1} in the span
            const bool lost = !dependent && !(p2 > 0.0);            // G no longer positive definite
            if (dependent) p2 = fmax(1e-30 * gjj, 1e-200);
            int act, k = j + 1;
            bool settled = false;
            if (!finite) {
                act = ACT_FAIL;
            } else if (lost) {
                act = ACT_UPDATE_CHECK;
                k = j;                                             // without the column that failed
            } else {
                const double pinv = rsqrt(p2);
                double* wn = tm + tri(j + 1);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int l = lane + 32 * h;
                    if (l <= j) {
                        double a[4] = {0.0, 0.0, 0.0, 0.0};
                        int i = l, at = tri(l) + l;
                        for (; i + 3 <= j; i += 4) {
#pragma unroll
                            for (int t = 0; t < 4; ++t) {
                                a[t] += vd[i + t] * tm[at];
                                at += i + t + 1;
                            }
                        }
                        for (; i <= j; ++i) {
                            a[0] += vd[i] * tm[at];
                            at += i + 1;
                        }
                        wn[l] = -((a[0] + a[1]) + (a[2] + a[3])) * pinv;
                    }
                }
                const double zn = (tj - s2[1]) * pinv;
                const double sz = ctl.sz + zn * zn;                // the residual estimate is 1 / sqrt(sz)
                const double stop = ctl.atol_eff, rest = kSettled<T> * ctl.bnorm;
                __syncwarp();
                if (lane == 0) {
                    wn[j + 1] = pinv;
                    va[j + 1] = zn;
                    vb[j + 1] = tj;
                    ctl.sz = sz;
                }
                settled = I.full_cycles && sz * rest * rest >= 1.0;
                if (!isfinite(zn)) act = ACT_FAIL;
                else if (!I.full_cycles && sz * stop * stop >= 1.0 && !dependent) act = ACT_UPDATE_FINAL;
                else if (j + 1 >= cycle_cols || dependent || settled) act = ACT_UPDATE_CHECK;
                else act = ACT_NEXT_J;
                __syncwarp();
            }
            if (act == ACT_UPDATE_FINAL || act == ACT_UPDATE_CHECK) {
                // residual coefficients c = W^T z / ||z||^2 over K_0..K_k
                const double isz = 1.0 / ctl.sz;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int l = lane + 32 * h;
                    if (l <= k) {
                        double a = 0.0;
                        for (int i = l; i <= k; ++i) a += tm[tri(i) + l] * va[i];
                        vc[l] = a * isz;
                    }
                }
                __syncwarp();
                // sum c_i K_i = r0 - A sum y_i K_i with A K_0 = theta K_0 + delta K_1,
                // A K_i = theta K_i + delta/2 (K_{i+1} + K_{i-1}): rows k..1 give y
                if (lane == 0) {
                    double y1 = 0.0, y2 = 0.0;      // y_i, y_{i+1}
                    for (int i = k; i >= 1; --i) {
                        const double y0 = -(vc[i] + I.theta * y1 + 0.5 * I.delta * y2) *
                                          (i == 1 ? I.inv_delta : 2.0 * I.inv_delta);
                        shc[i - 1] = y0;
                        y2 = y1;
                        y1 = y0;
                    }
                }
            }
            if (lane == 0) {
                ctl.action = act;
                ctl.k = k;
                ctl.settled = settled ? 1 : 0;
                if (act == ACT_FAIL) fail();
            }
        }
        decided();
    };
    // Arnoldi, phase A of column j: h_ij = s_i <V_i, w> and the coefficients
    // h_ij s_i that phase C subtracts
    auto decide_dots = [&](int j) {
        for (int i = threadIdx.x; i <= j; i += kThreads) {
            const double si = vb[i];
            const double h = si * gsum[i];
            vc[i] = h;
            shc[i] = h * si;
        }
        decided();
    };
    // Arnoldi, phase C of column j: Givens update of the Hessenberg column and,
    // when the cycle ends, the back substitution R y = g (g in va, s in vb,
    // the rotations in gv_cs and vd, the column in vc)
    __shared__ double gv_cs[kMaxRestart];
    auto decide_norm = [&](int j) {
        if (threadIdx.x == 0) {
            const double hn = sqrt(gsum[0]);
            vc[j + 1] = hn;
            for (int i = 0; i < j; ++i) {
                const double c = gv_cs[i], s = vd[i];
                const double a = vc[i], bb = vc[i + 1];
                vc[i] = c * a + s * bb;
                vc[i + 1] = -s * a + c * bb;
            }
            const double a = vc[j], bb = vc[j + 1];
            const double r = hypot(a, bb);
            const double c = (r == 0.0) ? 1.0 : a / r;
            const double s = (r == 0.0) ? 0.0 : bb / r;
            gv_cs[j] = c;
            vd[j] = s;
            vc[j] = r;
            for (int i = 0; i <= j; ++i) tm[tri(j) + i] = vc[i];
            const double gj = va[j];
            va[j] = c * gj;
            va[j + 1] = -s * gj;
            const double est = fabs(va[j + 1]);
            const bool breakdown = (hn == 0.0);
            const bool conv = (!I.full_cycles) && (est <= ctl.atol_eff);
            const bool settled = I.full_cycles && est <= kSettled<T> * ctl.bnorm;
            int act;
            if (!isfinite(hn) || !isfinite(r)) {
                act = ACT_FAIL;
            } else if (conv || (breakdown && !I.full_cycles)) {
                act = ACT_UPDATE_FINAL;
            } else if (j + 1 >= I.m || breakdown || settled) {
                act = ACT_UPDATE_CHECK;
            } else {
                act = ACT_NEXT_J;
                vb[j + 1] = 1.0 / hn;
                ctl.sj = vb[j + 1];
            }
            ctl.action = act;
            ctl.k = j + 1;
            ctl.settled = 1;    // nothing is left of the cycle
            if (act == ACT_FAIL) fail();
        }
        csync<ST>();
        if ((ctl.action == ACT_UPDATE_FINAL || ctl.action == ACT_UPDATE_CHECK) && warp == 0) {
            const int k = j + 1;
            for (int i = k - 1; i >= 0; --i) {
                double acc = 0.0;
                for (int l = i + 1 + lane; l < k; l += 32) acc += tm[tri(l) + i] * vc[l];
                acc = warp_sum(acc);
                if (lane == 0) vc[i] = (va[i] - acc) / tm[tri(i) + i];
                __syncwarp();
            }
            // x += sum_j y_j v_j = sum_j (y_j s_j) V_j
            for (int i = lane; i < k; i += 32) shc[i] = vc[i] * vb[i];
        }
        decided();
    };
    auto decide_check = [&]() {
        // columns the logical cycle of I.m still has: when its Gram matrix gave out
        // early, or once more when it ended settled (kRefine)
        const int left = I.m - cols;
        const bool basis = cheb && ctl.cheb;
        const double rn = sqrt(gsum[0]);
        const bool more = basis && I.full_cycles && left > 0 && rn > kRefine<T> * ctl.bnorm && !ctl.refined;
        csync<ST>();
        if (threadIdx.x == 0) {
            // early exit, the Gram matrix gave out: such a short cycle is not one of those
            // that maxiter counts (m columns each), so the solve has as many whole cycles
            // as Arnoldi's would, from a smaller residual.  The form stays while short
            // cycles halve the residual and add up to less than maxiter columns (one pass
            // per column: 64 x 64 sheet, plane front, half width 60, restart 20, tol 1e-5:
            // 44 passes per solve, 67 with Arnoldi from the first short cycle on)
            if (more) {
                if (ctl.settled) ctl.refined = 1;
            } else if (basis && !I.full_cycles && left > 0) {
                ctl.iters_short += cols;
                if (ctl.iters_short >= I.maxiter || rn > 0.5 * ctl.rnorm) ctl.cheb = 0;
            } else {
                ctl.iters_cap += I.m;
                ctl.refined = 0;
            }
            if (gsum[0] < kTinySquare) ctl.cheb = 0;
            if (!isfinite(rn)) {
                fail();
            } else if (more) {
                start_cycle(gsum[0]);
            } else if (rn <= ctl.atol_eff) {
                ctl.action = ACT_DONE;
            } else if (ctl.iters_cap >= I.maxiter) {
                ctl.action = ACT_DONE;
                st_nonconv += 1;
                if (rank == 0 && I.st->status == PHS_OK) I.st->status = PHS_WARN_NO_CONVERGE;
            } else {
                start_cycle(gsum[0]);
            }
        }
        decided();
        if (!more) cols = 0;
        if (ctl.action == ACT_DONE) account_solve();
    };

    // ---- sample / activation bookkeeping of the state in u (after step s-1)
    auto sample_voxel = [&](long long n, T un, T hn, long long done_step) {
        if (pending >= 0) {
            I.hist_u[(size_t)pending * N + n] = un;
            if (I.save_h) I.hist_h[(size_t)pending * N + n] = hn;
        }
        if (done_step >= 0 && un >= T(0.5) && I.lat[n] < 0) I.lat[n] = (int32_t)done_step;
    };

    // End-of-step work of voxel n whose new state un is known (the state after
    // step done_step): its sample into history slot `slot` (-1: none), its
    // activation entry (lat_n loaded when un >= 0.5), then the RK4 reaction of
    // the next step (stimulus bits stim_next) -> h of the step after it into
    // hdst, u* returned.  This is the reaction pass of the next step, done while
    // the voxel's new state is still in registers.
    auto react_voxel = [&](long long n, T un, T hn, int32_t lat_n, long long done_step, int slot, uint8_t fl,
                           uint8_t stim_next, T* hdst) -> T {
        if (slot >= 0) {
            I.hist_u[(size_t)slot * N + n] = un;
            if (I.save_h) I.hist_h[(size_t)slot * N + n] = hn;
        }
        if (done_step >= 0 && un >= T(0.5) && lat_n < 0) I.lat[n] = (int32_t)done_step;
        T p[5];
        params_of(n, p);
        const T J = (fl & stim_next & 3u) ? I.jmag : T(0);
        T us, hs;
        rk4(I.model, un, hn, J, p, I.dt, us, hs);
        hdst[n] = hs;
        return us;
    };

    // the reaction pass of the current step was done at the end of the previous
    // one (by the same threads, for the same voxels)
    bool prepared = false;
    for (; step < step_end && !retired && !aborted; ++step) {
        const uint8_t stim_bits = __ldg(I.stim + step);
        const bool tb = step < I.tb_steps;
        T* hin = hbuf ? I.h1 : I.h0;
        T* hout = hbuf ? I.h0 : I.h1;

        // ================= RHS phase.  Pass 1: RK4 reaction of every voxel of the
        // team, u* into the pairs.  Except in the first step of a launch and after
        // a full-cycle solve, it ran at the end of the previous step (react_voxel
        // in the update and copy passes), so it costs no pass of its own.
        // Pass 2, after a team barrier: b = u* + dt/2 L u*, the initial guess
        // x0 = u* + dx and r0 = b - A x0 -> V0.  u* and the increment dx lie side by
        // side, so one gather per neighbour brings both; x0 and b are not stored
        // (x0 is u* + dx again in the update; only full cycles read b).
        for (int grp = prepared ? n_groups : rank; grp < n_groups; grp += P) {
            for (int tile = grp * gt; tile < min(n_tiles, (grp + 1) * gt); ++tile) {
                // every load of the tile before its first store: plain loads cannot
                // move across stores the compiler must assume may alias them
                T un[VPT], hn[VPT];
                uint8_t fl[VPT];
                int32_t lt[VPT];
#pragma unroll
                for (int v = 0; v < VPT; ++v) {
                    const long long n = voxel(tile, v);
                    un[v] = I.u[n];
                    hn[v] = hin[n];
                    fl[v] = __ldg(I.vflags + n);
                }
#pragma unroll
                for (int v = 0; v < VPT; ++v)
                    lt[v] = (step > 0 && un[v] >= T(0.5)) ? I.lat[voxel(tile, v)] : 0;
#pragma unroll
                for (int v = 0; v < VPT; ++v) {
                    const long long n = voxel(tile, v);
                    if (n < N) UD[n].x = react_voxel(n, un[v], hn[v], lt[v], step - 1, pending, fl[v], stim_bits, hout);
                }
            }
        }
        pending = -1;
        mark(PF_RHS1);
        if (!barrier()) { aborted = true; break; }
        mark(PF_RHS_WAIT);
        phase_begin();
        for (int grp = rank; grp < n_groups; grp += P) {
            for (int tile = grp * gt; tile < min(n_tiles, (grp + 1) * gt); ++tile) {
                if (pf_on && lane == 0) {
                    const int nxt = tile_after(grp, tile);
                    if (warp < kRowArrays) pf_rows(warp, nxt);
                    else if (warp == kRowArrays) pf_slice(UD, sizeof(P2), nxt);
                }
                const long long n0 = voxel(tile, 0);
                P2 own[VPT], lap[VPT];
#pragma unroll
                for (int v = 0; v < VPT; ++v) own[v] = UD[n0 + v * kThreads];
                tile_lap<T, VPT, EDGE, NB>(I, UD, n0, tb, own, lap);
                double s[2] = {0.0, 0.0};
#pragma unroll
                for (int v = 0; v < VPT; ++v) {
                    const long long n = n0 + v * kThreads;
                    const T x0 = own[v].x + own[v].y;
                    const T bn = own[v].x + I.half_dt * lap[v].x;
                    const T ax = x0 - I.half_dt * (lap[v].x + lap[v].y);
                    const T rn = bn - ax;
                    if (I.full_cycles) I.b[n] = bn;
                    Vb[n] = rn;
                    s[0] += (double)bn * (double)bn;
                    s[1] += (double)rn * (double)rn;
                }
                const double w = warp_sums<2>(s, lane);
                if ((lane & 15) == 0) put(2, lane >> 4, w, tile == grp * gt);
            }
            group_done(2);
        }
        mark(PF_RHS);
        if (!barrier_sums(2)) { aborted = true; break; }
        iters_solve = 0;
        cols = 0;
        decide_rhs();
        int act = ctl.action;
        mark(PF_RHS_WAIT);
        // end of this step: its history slot, and whether the pass that writes
        // the new state also runs the next step's reaction (not after the last
        // step of the launch)
        const bool due_now = (I.stride > 0) ? (step % I.stride == 0) : true;
        const int slot_now = (due_now && id_save < I.n_samples) ? id_save : -1;
        const bool fuse_next = step + 1 < step_end;
        const uint8_t stim_next = fuse_next ? __ldg(I.stim + step + 1) : (uint8_t)0;
        bool fused = false;

        if (act == ACT_CYCLE) {
            bool first_cycle = true;
            for (;;) {
                if (cheb && ctl.cheb) {
                    const int cycle_cols = I.m - cols;
                    for (int j = 0;; ++j) {
                        // ======== column j: K_{j+1} = 2/delta (A - theta) K_j - K_{j-1}, dots
                        const T* Kj = Vb + (size_t)j * ldV;
                        const T* Kp = Vb + (size_t)max(j - 1, 0) * ldV;
                        T* Kn = Vb + (size_t)(j + 1) * ldV;
                        const int ns = j + 2;
                        const T ca = (j == 0) ? I.cheb_a : T(2) * I.cheb_a;   // (1 - theta)/delta, doubled
                        const T cb = (j == 0) ? I.cheb_b : T(2) * I.cheb_b;   // -dt/2 / delta, doubled
                        const T cc = (j == 0) ? T(0) : T(1);
                        phase_begin();
                        for (int grp = rank; grp < n_groups; grp += P) {
                            for (int tile = grp * gt; tile < min(n_tiles, (grp + 1) * gt); ++tile) {
                                if (pf_on && lane < 1 + (kRowArrays + j) / kWarps) {
                                    const int nxt = tile_after(grp, tile), id = warp + kWarps * lane;
                                    if (id < kRowArrays) pf_rows(id, nxt);
                                    else if (id <= kRowArrays + j)
                                        pf_slice(Vb + (size_t)(id - kRowArrays) * ldV, sizeof(T), nxt);
                                }
                                const bool first = tile == grp * gt;
                                const long long n0 = voxel(tile, 0);
                                T own[VPT], lap[VPT], prev[VPT], kn[VPT];
                                T vv[kChunk][VPT];      // K_{j-2}, K_{j-3}, ... (in the slots 3.. of the first sums)
#pragma unroll
                                for (int v = 0; v < VPT; ++v) {
                                    own[v] = Kj[n0 + v * kThreads];
                                    prev[v] = Kp[n0 + v * kThreads];
                                }
#pragma unroll
                                for (int e = 3; e < kChunk; ++e)
#pragma unroll
                                    for (int v = 0; v < VPT; ++v)
                                        vv[e][v] = (j + 1 >= e) ? Vb[(size_t)(j + 1 - e) * ldV + n0 + v * kThreads] : T(0);
                                tile_lap<T, VPT, EDGE, NB>(I, Kj, n0, tb, own, lap);
#pragma unroll
                                for (int v = 0; v < VPT; ++v) {
                                    kn[v] = (ca * own[v] + cb * lap[v]) - cc * prev[v];
                                    vv[0][v] = kn[v];
                                    vv[1][v] = own[v];
                                    vv[2][v] = prev[v];
                                }
                                double s[kChunk];
#pragma unroll
                                for (int e = 0; e < kChunk; ++e) {
                                    s[e] = 0.0;
#pragma unroll
                                    for (int v = 0; v < VPT; ++v) s[e] += (double)vv[e][v] * (double)kn[v];
                                }
                                {
                                    const double w = warp_sums<kChunk>(s, lane);
                                    const int i = j + 1 - (lane >> (5 - log2_of(kChunk)));
                                    if ((lane & (32 / kChunk - 1)) == 0 && i >= 0) put(ns, i, w, first);
                                }
                                for (int i0 = j + 1 - kChunk; i0 >= 0; i0 -= kChunk) {   // K_{i0}, K_{i0-1}, ...
#pragma unroll
                                    for (int e = 0; e < kChunk; ++e)
#pragma unroll
                                        for (int v = 0; v < VPT; ++v)
                                            vv[e][v] = (i0 >= e) ? Vb[(size_t)(i0 - e) * ldV + n0 + v * kThreads] : T(0);
#pragma unroll
                                    for (int e = 0; e < kChunk; ++e) {
                                        s[e] = 0.0;
#pragma unroll
                                        for (int v = 0; v < VPT; ++v) s[e] += (double)vv[e][v] * (double)kn[v];
                                    }
                                    const double w = warp_sums<kChunk>(s, lane);
                                    const int i = i0 - (lane >> (5 - log2_of(kChunk)));
                                    if ((lane & (32 / kChunk - 1)) == 0 && i >= 0) put(ns, i, w, first);
                                }
#pragma unroll
                                for (int v = 0; v < VPT; ++v) Kn[n0 + v * kThreads] = kn[v];
                            }
                            group_done(ns);
                        }
                        mark(PF_A);
                        if (!barrier_sums(ns)) { aborted = true; break; }
                        iters_solve += 1;
                        cols += 1;
                        decide_cheb(j, cycle_cols);
                        act = ctl.action;
                        mark(PF_A_WAIT);
                        if (prof_on && threadIdx.x == 0) pf[PF_SOLVE_ITERS] += 1;
                        if (act != ACT_NEXT_J) break;
                    }
                } else {
                    for (int j = 0;; ++j) {
                        // ======== phase A: w = A (s_j V_j) -> V_{j+1}; dots <V_i, w>
                        const T sj = (T)ctl.sj;
                        const T* Vj = Vb + (size_t)j * ldV;
                        T* Vn = Vb + (size_t)(j + 1) * ldV;
                        const int ns = j + 1;
                        phase_begin();
                        for (int grp = rank; grp < n_groups; grp += P) {
                            for (int tile = grp * gt; tile < min(n_tiles, (grp + 1) * gt); ++tile) {
                                const bool first = tile == grp * gt;
                                const long long n0 = voxel(tile, 0);
                                T own[VPT], lap[VPT], wr[VPT];
#pragma unroll
                                for (int v = 0; v < VPT; ++v) own[v] = Vj[n0 + v * kThreads];
                                tile_lap<T, VPT, EDGE, NB>(I, Vj, n0, tb, own, lap);
#pragma unroll
                                for (int v = 0; v < VPT; ++v) wr[v] = sj * (own[v] - I.half_dt * lap[v]);
                                for (int i0 = 0; i0 <= j; i0 += kChunk) {
                                    T vv[kChunk][VPT];
                                    double s[kChunk];
#pragma unroll
                                    for (int e = 0; e < kChunk; ++e)
#pragma unroll
                                        for (int v = 0; v < VPT; ++v)
                                            vv[e][v] = (i0 + e <= j) ? Vb[(size_t)(i0 + e) * ldV + n0 + v * kThreads] : T(0);
#pragma unroll
                                    for (int e = 0; e < kChunk; ++e) {
                                        s[e] = 0.0;
#pragma unroll
                                        for (int v = 0; v < VPT; ++v) s[e] += (double)vv[e][v] * (double)wr[v];
                                    }
                                    const double w = warp_sums<kChunk>(s, lane);
                                    const int i = i0 + (lane >> (5 - log2_of(kChunk)));
                                    if ((lane & (32 / kChunk - 1)) == 0 && i <= j) put(ns, i, w, first);
                                }
#pragma unroll
                                for (int v = 0; v < VPT; ++v) Vn[n0 + v * kThreads] = wr[v];
                            }
                            group_done(ns);
                        }
                        mark(PF_A);
                        if (!barrier_sums(ns)) { aborted = true; break; }
                        decide_dots(j);
                        mark(PF_A_WAIT);
                        // ======== phase C: u = w - sum_i c_i V_i  (in place), ||u||^2
                        phase_begin();
                        for (int grp = rank; grp < n_groups; grp += P) {
                            for (int tile = grp * gt; tile < min(n_tiles, (grp + 1) * gt); ++tile) {
                                const long long n0 = voxel(tile, 0);
                                double acc[VPT], s[1] = {0.0};
#pragma unroll
                                for (int v = 0; v < VPT; ++v) acc[v] = (double)Vn[n0 + v * kThreads];
                                for (int i0 = 0; i0 <= j; i0 += kChunk) {
                                    T vv[kChunk][VPT];
#pragma unroll
                                    for (int e = 0; e < kChunk; ++e)
#pragma unroll
                                        for (int v = 0; v < VPT; ++v)
                                            vv[e][v] = (i0 + e <= j) ? Vb[(size_t)(i0 + e) * ldV + n0 + v * kThreads] : T(0);
#pragma unroll
                                    for (int e = 0; e < kChunk; ++e) {
                                        const double cf = (i0 + e <= j) ? shc[i0 + e] : 0.0;
#pragma unroll
                                        for (int v = 0; v < VPT; ++v) acc[v] -= cf * (double)vv[e][v];
                                    }
                                }
#pragma unroll
                                for (int v = 0; v < VPT; ++v) {
                                    const T ut = (T)acc[v];
                                    Vn[n0 + v * kThreads] = ut;
                                    s[0] += (double)ut * (double)ut;
                                }
                                const double w = warp_sums<1>(s, lane);
                                if (lane == 0) put(1, 0, w, tile == grp * gt);
                            }
                            group_done(1);
                        }
                        mark(PF_C);
                        if (!barrier_sums(1)) { aborted = true; break; }
                        iters_solve += 1;
                        decide_norm(j);
                        act = ctl.action;
                        mark(PF_C_WAIT);
                        if (prof_on && threadIdx.x == 0) pf[PF_SOLVE_ITERS] += 1;
                        if (act != ACT_NEXT_J) break;
                    }
                }
                if (aborted) break;
                if (act == ACT_FAIL) { retired = true; break; }
                // ============ phase X: x += sum_j c_j V_j
                const int k = ctl.k;
                const bool final = (act == ACT_UPDATE_FINAL);
                const bool react = final && fuse_next;
                if (final) account_solve();
                int nsx = 0;
                if constexpr (ST) {
                    stg.begin();
                    const int o_ud = stg.add(UD, sizeof(P2));
                    const int o_x = first_cycle ? -1 : stg.add(I.x, sizeof(T));
                    const int o_h = react ? stg.add(hout, sizeof(T)) : -1;
                    const int o_fl = react ? stg.add(I.vflags, 1) : -1;
                    const int nvs = min(k, stg.vec_cap());
                    const int o_v = stg.lay_off;
                    for (int i = 0; i < nvs; ++i) stg.add(Vb + (size_t)i * ldV, sizeof(T));
                    nsx = stg.publish(rank, P, n_tiles, n_groups, gt);
                    for (int grp = rank; nsx > 0 && grp < n_groups; grp += P) {
                        for (int tile = grp * gt; tile < min(n_tiles, (grp + 1) * gt); ++tile) {
                            const unsigned char* sb = stg.acquire(abort_word);
                            double acc[VPT];
                            T x0[VPT], dxo[VPT], hn[VPT];
                            uint8_t fl[VPT];
                            int32_t lt[VPT];
#pragma unroll
                            for (int v = 0; v < VPT; ++v) {
                                const int li = v * kThreads + threadIdx.x;
                                const P2 p = reinterpret_cast<const P2*>(sb + o_ud)[li];
                                dxo[v] = p.y;
                                x0[v] = first_cycle ? p.x + p.y : reinterpret_cast<const T*>(sb + o_x)[li];
                                acc[v] = (double)x0[v];
                                hn[v] = react ? reinterpret_cast<const T*>(sb + o_h)[li] : T(0);
                                fl[v] = react ? sb[o_fl + li] : (uint8_t)0;
                            }
                            for (int i = 0; i < k; ++i) {
                                const double cf = shc[i];
#pragma unroll
                                for (int v = 0; v < VPT; ++v) {
                                    const int li = v * kThreads + threadIdx.x;
                                    const T val = (i < nvs) ? reinterpret_cast<const T*>(sb + o_v + i * TILE * (int)sizeof(T))[li]
                                                            : Vb[(size_t)i * ldV + (long long)tile * TILE + li];
                                    acc[v] += cf * (double)val;
                                }
                            }
                            stg.release();
#pragma unroll
                            for (int v = 0; v < VPT; ++v)
                                lt[v] = (react && (T)acc[v] >= T(0.5)) ? I.lat[voxel(tile, v)] : 0;
#pragma unroll
                            for (int v = 0; v < VPT; ++v) {
                                const long long n = voxel(tile, v);
                                if (n >= N) continue;
                                const T un = (T)acc[v];
                                if (!final) {
                                    I.x[n] = un;
                                    continue;
                                }
                                I.u[n] = un;
                                const T dx = I.guess ? (T)((double)dxo[v] + (acc[v] - (double)x0[v])) : T(0);
                                if (react) {
                                    P2 p;
                                    p.x = react_voxel(n, un, hn[v], lt[v], step, slot_now, fl[v], stim_next, hin);
                                    p.y = dx;
                                    UD[n] = p;
                                } else {
                                    UD[n].y = dx;
                                }
                            }
                        }
                    }
                }
                for (int grp = rank; nsx == 0 && grp < n_groups; grp += P) {
                    for (int tile = grp * gt; tile < min(n_tiles, (grp + 1) * gt); ++tile) {
                        if (pf_on && lane < 1 + (k + 2) / kWarps) {
                            const int nxt = tile_after(grp, tile), id = warp + kWarps * lane;
                            if (id < k) pf_slice(Vb + (size_t)id * ldV, sizeof(T), nxt);
                            else if (id == k) pf_slice(UD, sizeof(P2), nxt);
                            else if (id == k + 1 && react) pf_slice(hout, sizeof(T), nxt);
                            else if (id == k + 2 && react) pf_slice(I.vflags, 1, nxt);
                        }
                        double acc[VPT];
                        T x0[VPT], dxo[VPT], hn[VPT];
                        uint8_t fl[VPT];
                        int32_t lt[VPT];
#pragma unroll
                        for (int v = 0; v < VPT; ++v) {
                            const long long n = voxel(tile, v);
                            const P2 p = UD[n];
                            dxo[v] = p.y;
                            x0[v] = first_cycle ? p.x + p.y : I.x[n];
                            acc[v] = (double)x0[v];
                            hn[v] = react ? hout[n] : T(0);
                            fl[v] = react ? __ldg(I.vflags + n) : (uint8_t)0;
                        }
                        // kChunk vectors' loads at a time
                        for (int i0 = 0; i0 < k; i0 += kChunk) {
                            T vv[kChunk][VPT];
#pragma unroll
                            for (int e = 0; e < kChunk; ++e)
#pragma unroll
                                for (int v = 0; v < VPT; ++v)
                                    vv[e][v] = (i0 + e < k) ? Vb[(size_t)(i0 + e) * ldV + voxel(tile, v)] : T(0);
#pragma unroll
                            for (int e = 0; e < kChunk; ++e) {
                                if (i0 + e < k) {
                                    const double cf = shc[i0 + e];
#pragma unroll
                                    for (int v = 0; v < VPT; ++v) acc[v] += cf * (double)vv[e][v];
                                }
                            }
                        }
#pragma unroll
                        for (int v = 0; v < VPT; ++v)
                            lt[v] = (react && (T)acc[v] >= T(0.5)) ? I.lat[voxel(tile, v)] : 0;
#pragma unroll
                        for (int v = 0; v < VPT; ++v) {
                            const long long n = voxel(tile, v);
                            if (n >= N) continue;
                            const T un = (T)acc[v];
                            if (!final) {
                                I.x[n] = un;
                                continue;
                            }
                            I.u[n] = un;
                            // increment u_next - u* for the next step's initial guess
                            const T dx = I.guess ? (T)((double)dxo[v] + (acc[v] - (double)x0[v])) : T(0);
                            if (react) {
                                P2 p;
                                p.x = react_voxel(n, un, hn[v], lt[v], step, slot_now, fl[v], stim_next, hin);
                                p.y = dx;
                                UD[n] = p;
                            } else {
                                UD[n].y = dx;
                            }
                        }
                    }
                }
                mark(PF_X);
                if (final) {
                    fused = react;
                    break;
                }
                first_cycle = false;
                // ============ true residual of the new iterate (start of the next cycle)
                if (!barrier()) { aborted = true; break; }
                phase_begin();
                for (int grp = rank; grp < n_groups; grp += P) {
                    for (int tile = grp * gt; tile < min(n_tiles, (grp + 1) * gt); ++tile) {
                        const long long n0 = voxel(tile, 0);
                        T own[VPT], lap[VPT], bn[VPT];
#pragma unroll
                        for (int v = 0; v < VPT; ++v) own[v] = I.x[n0 + v * kThreads];
                        if (I.full_cycles) {
#pragma unroll
                            for (int v = 0; v < VPT; ++v) bn[v] = I.b[n0 + v * kThreads];
                        } else {
                            // b again from u* (the pairs are untouched until the solve ends)
                            P2 po[VPT], pl[VPT];
#pragma unroll
                            for (int v = 0; v < VPT; ++v) po[v] = UD[n0 + v * kThreads];
                            tile_lap<T, VPT, EDGE, NB>(I, UD, n0, tb, po, pl);
#pragma unroll
                            for (int v = 0; v < VPT; ++v) bn[v] = po[v].x + I.half_dt * pl[v].x;
                        }
                        tile_lap<T, VPT, EDGE, NB>(I, I.x, n0, tb, own, lap);
                        double s[1] = {0.0};
#pragma unroll
                        for (int v = 0; v < VPT; ++v) {
                            const long long n = n0 + v * kThreads;
                            const T r = bn[v] - (own[v] - I.half_dt * lap[v]);
                            Vb[n] = r;
                            if (n < N) I.u[n] = own[v];
                            s[0] += (double)r * (double)r;
                        }
                        const double w = warp_sums<1>(s, lane);
                        if (lane == 0) put(1, 0, w, tile == grp * gt);
                    }
                    group_done(1);
                }
                mark(PF_CHECK);
                if (!barrier_sums(1)) { aborted = true; break; }
                decide_check();
                act = ctl.action;
                mark(PF_CHECK_WAIT);
                if (act == ACT_DONE) break;
                if (act == ACT_FAIL) { retired = true; break; }
                // ACT_CYCLE: V0 holds the new residual
            }
            if (aborted || retired) break;
        } else if (act == ACT_ZERO_B || act == ACT_DONE) {
            // no iteration: the solve returns x0 (or b = 0)
            for (int grp = rank; grp < n_groups; grp += P) {
                for (int tile = grp * gt; tile < min(n_tiles, (grp + 1) * gt); ++tile) {
                    if (pf_on && lane == 0 && warp < 3) {
                        const int nxt = tile_after(grp, tile);
                        if (warp == 0) pf_slice(UD, sizeof(P2), nxt);
                        else if (warp == 1 && fuse_next) pf_slice(hout, sizeof(T), nxt);
                        else if (warp == 2 && fuse_next) pf_slice(I.vflags, 1, nxt);
                    }
                    T un[VPT], dxo[VPT], hn[VPT];
                    uint8_t fl[VPT];
                    int32_t lt[VPT];
#pragma unroll
                    for (int v = 0; v < VPT; ++v) {
                        const long long n = voxel(tile, v);
                        const P2 p = UD[n];
                        dxo[v] = p.y;
                        un[v] = (act == ACT_ZERO_B) ? T(0) : p.x + p.y;
                        hn[v] = fuse_next ? hout[n] : T(0);
                        fl[v] = fuse_next ? __ldg(I.vflags + n) : (uint8_t)0;
                    }
#pragma unroll
                    for (int v = 0; v < VPT; ++v)
                        lt[v] = (fuse_next && un[v] >= T(0.5)) ? I.lat[voxel(tile, v)] : 0;
#pragma unroll
                    for (int v = 0; v < VPT; ++v) {
                        const long long n = voxel(tile, v);
                        if (n >= N) continue;
                        I.u[n] = un[v];
                        if (fuse_next) {
                            P2 p;
                            p.x = react_voxel(n, un[v], hn[v], lt[v], step, slot_now, fl[v], stim_next, hin);
                            p.y = dxo[v];
                            UD[n] = p;
                        }
                    }
                }
            }
            fused = fuse_next;
        } else {  // ACT_FAIL
            retired = true;
            break;
        }
        mark(PF_COPY);
        // No barrier at the end of the step: each voxel's u, h and pair are written
        // and read again (next RHS pass 1) by the same thread, and every cross-CTA
        // read of the next step follows its mid-RHS barrier.
        if (prof_on && threadIdx.x == 0) pf[PF_STEPS] += 1;
        hbuf ^= 1;
        if (slot_now >= 0) {
            ++id_save;
            pending = fused ? -1 : slot_now;    // a fused pass wrote the sample already
        }
        prepared = fused;
    }

    // flush the sample and activation test of the last completed step
    if (!aborted && !retired) {
        const T* hcur = hbuf ? I.h1 : I.h0;
        if (pending >= 0 || step > sh_step0) {
            for (int grp = rank; grp < n_groups; grp += P)
                for (int tile = grp * gt; tile < min(n_tiles, (grp + 1) * gt); ++tile) {
#pragma unroll
                    for (int v = 0; v < VPT; ++v) {
                        const long long n = voxel(tile, v);
                        if (n < N) sample_voxel(n, I.u[n], hcur[n], step - 1);
                    }
                }
        }
        pending = -1;
    }
    if (prof_on && threadIdx.x == 0) {
        for (int i = 0; i < kProfSlots; ++i)
            if (i != PF_TEAM) atomicAdd(I.prof + i, pf[i]);
        atomicExch(I.prof + PF_TEAM, (unsigned long long)P);
    }
    if (threadIdx.x == 0 && !aborted) {
        InstState* st = I.st;
        if (rank == 0) {
            st->arnoldi += st_arnoldi;
            st->arnoldi_sq += st_arnoldi_sq;
            st->solves += st_solves;
            if (st_max_arnoldi > st->max_arnoldi) st->max_arnoldi = st_max_arnoldi;
            st->nonconv += st_nonconv;
        }
        // the last CTA to leave records the progress and clears the counters: every
        // CTA has passed its last poll by then
        cuda::atomic_ref<unsigned int, cuda::thread_scope_device> ex(I.sync->exits);
        if (ex.fetch_add(1u, cuda::memory_order_acq_rel) == (unsigned int)(P - 1)) {
            st->step = step;
            st->id_save = id_save;
            st->pending = pending;
            st->hbuf = hbuf;
            I.sync->count = 0u;
            I.sync->exits = 0u;
        }
    }
    if constexpr (ST) stg.quit();   // the producer warp drains its copies and exits
}

// ------------------------------------------------------------------ fill kernel
template <typename T>
__global__ void fill_kernel(T* p, long long n, T v) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long s = (long long)gridDim.x * blockDim.x;
    for (; i < n; i += s) p[i] = v;
}

template <typename T>
__global__ void convert_kernel(const double* src, T* dst, long long n) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long s = (long long)gridDim.x * blockDim.x;
    for (; i < n; i += s) dst[i] = (T)src[i];
}

}  // namespace phs

// ====================================================================== host side
using namespace phs;

namespace {

constexpr int kVptF32 = 4;
constexpr int kVptF32Min = 2;    // the smallest voxels-per-thread of any FP32 variant
constexpr int kVptF64 = 1;

// Compiled step-kernel variants: the same algorithm with different tile
// lengths (voxels per thread; a tile is 256 x VPT consecutive voxels),
// register budgets (__launch_bounds__ minimum CTAs per SM), neighbour tables
// (int32 or compact) and, for the FP32 staged ones, the shared-memory ring of
// the producer warp (bytes; sized so that MINB CTAs fit an SM next to the
// kernel's static shared memory).  The autotuner picks one.  Each exists
// without and with the anisotropic edge terms.
using StepFnF = void (*)(const InstDev<float>*, const int4*, long long, unsigned int*);
using StepFnD = void (*)(const InstDev<double>*, const int4*, long long, unsigned int*);
constexpr int kRing3 = 48 * 1024, kRing2 = 84 * 1024;
const StepFnF kStepF32[] = {step_kernel<float, kVptF32, 2, false, 0, false>, step_kernel<float, kVptF32, 3, false, 0, false>,
                            step_kernel<float, kVptF32, 4, false, 0, false>, step_kernel<float, 2, 4, false, 0, false>,
                            step_kernel<float, 2, 5, false, 0, false>,       step_kernel<float, 2, 3, false, kRing3, false>,
                            step_kernel<float, 4, 2, false, kRing2, false>,  step_kernel<float, 2, 4, false, 0, true>,
                            step_kernel<float, kVptF32, 4, false, 0, true>};
const StepFnF kStepF32Edge[] = {step_kernel<float, kVptF32, 2, true, 0, false>, step_kernel<float, kVptF32, 3, true, 0, false>,
                                step_kernel<float, kVptF32, 4, true, 0, false>, step_kernel<float, 2, 4, true, 0, false>,
                                step_kernel<float, 2, 5, true, 0, false>,       step_kernel<float, 2, 3, true, kRing3, false>,
                                step_kernel<float, 4, 2, true, kRing2, false>,  step_kernel<float, 2, 4, true, 0, true>,
                                step_kernel<float, kVptF32, 4, true, 0, true>};
const int kMinbF32[] = {2, 3, 4, 4, 5, 3, 2, 4, 4};
const int kVptOfF32[] = {kVptF32, kVptF32, kVptF32, 2, 2, 2, 4, 2, kVptF32};
const int kRingF32[] = {0, 0, 0, 0, 0, kRing3, kRing2, 0, 0};
// variants that read the compact neighbour table of every instance, and their
// int32-table twin (launched instead when an unfinished instance has none)
const int kTwinF32[] = {-1, -1, -1, -1, -1, -1, -1, 3, 2};
const StepFnD kStepF64[] = {step_kernel<double, kVptF64, 2, false, 0, false>, step_kernel<double, kVptF64, 3, false, 0, false>};
const StepFnD kStepF64Edge[] = {step_kernel<double, kVptF64, 2, true, 0, false>,
                                step_kernel<double, kVptF64, 3, true, 0, false>};
const int kMinbF64[] = {2, 3};
constexpr int kNumF32 = 9, kNumF64 = 2;
// Threads per CTA and dynamic shared memory of a variant's launch.
int ring_of(int prec_bytes, int variant) { return prec_bytes == 8 ? 0 : kRingF32[variant]; }
int threads_of(int prec_bytes, int variant) { return kThreads + (ring_of(prec_bytes, variant) > 0 ? 32 : 0); }
int dyn_smem_of(int prec_bytes, int variant) {
    const int r = ring_of(prec_bytes, variant);
    return r > 0 ? kRingHeader + r : 0;
}

// Tiles of an instance of n voxels under a variant.
int tiles_of(long long n, int vpt) { return (int)((n + (long long)kThreads * vpt - 1) / ((long long)kThreads * vpt)); }
// Tiles per group of partial sums, and groups, of an instance of `tiles` tiles.
template <typename T>
int group_tiles(int tiles) {
    const int most = sizeof(T) == 8 ? kMaxGroupsF64 : kMaxGroupsF32;
    return std::max(1, (tiles + most - 1) / most);
}
template <typename T>
int groups_of(int tiles) {
    const int g = group_tiles<T>(tiles);
    return (tiles + g - 1) / g;
}
int vpt_of(int prec_bytes, int variant) { return prec_bytes == 8 ? kVptF64 : kVptOfF32[variant]; }
// FP32: 512-voxel tiles, 64 registers, 4 CTAs/SM, compact table: a lone
// instance spreads over twice the CTAs of 1024-voxel tiles (91k voxels: 6.5
// against 8.0 ms per 300 steps, 40k: 5.5 against 6.7 per 200) and a batch of
// 3.9M voxels takes the same (88-92 ms per 300 steps).  FP64: 80 registers, 3
// CTAs/SM (plain form, 160k voxels: 11.9 ms per 30 steps against 14.3 ms with
// 124 registers and 2 CTAs/SM).
constexpr int kDefaultF32 = 7, kDefaultF64 = 1;

template <typename T>
const void* step_fn(int variant, bool edge = false) {
    if (sizeof(T) == 8) return edge ? (const void*)kStepF64Edge[variant] : (const void*)kStepF64[variant];
    return edge ? (const void*)kStepF32Edge[variant] : (const void*)kStepF32[variant];
}

struct InstHost {
    bool used = false;
    bool finished = false;
    bool exported = false;       // u, hist_u and lat are allocations of their own (export_arrays)
    phs_instance_desc d{};
    long long n = 0;
    long long ldv = 0;           // padded voxel count: length of every per-voxel array
    int n_tiles = 0;
    int m = 0;
    void* nb = nullptr;
    int16_t* nbr = nullptr;      // compact neighbour table, or nullptr
    int32_t* nbase = nullptr;
    void* coef = nullptr;
    void* cw = nullptr;
    void* m6 = nullptr;
    void* enb = nullptr;
    void* ecf = nullptr;
    void* vflags = nullptr;
    void* vparams = nullptr;
    void* stim = nullptr;
    void* u = nullptr;
    void* h0 = nullptr;
    void* h1 = nullptr;
    void* x = nullptr;
    void* b = nullptr;
    void* V = nullptr;
    void* ud = nullptr;
    void* hist_u = nullptr;
    void* hist_h = nullptr;
    int32_t* lat = nullptr;
    double* part = nullptr;
    long long part_half = 0;
    double bound = 0.0;          // largest eigenvalue Gershgorin's theorem allows -L
    TeamSync* sync = nullptr;
    InstState* st = nullptr;
    unsigned long long* prof = nullptr;
    InstState st_host{};
    double kavg = 4.0;           // recent columns per step (cost model)
    long long ref_arnoldi = 0;   // counters at the last rebalance
    long long ref_step = 0;
    double weight = 0.0;         // measured CTA-time per step (0: use the model)
    int team = 0;                // CTAs given to this instance by the current plan
    unsigned long long prof_ref[16] = {};
};

// The engine's device for as long as the guard lives (an engine may be
// destroyed from a thread that has another device current).
struct DeviceGuard {
    int old = -1;
    explicit DeviceGuard(int device) {
        if (cudaGetDevice(&old) != cudaSuccess || old == device || cudaSetDevice(device) != cudaSuccess) old = -1;
    }
    ~DeviceGuard() {
        if (old >= 0) cudaSetDevice(old);
    }
};

void free_inst(InstHost& h) {
    if (h.exported) {
        cudaFree(h.u);
        cudaFree(h.hist_u);
        cudaFree(h.lat);
        h.u = h.hist_u = nullptr;
        h.lat = nullptr;
    }
    void* ptrs[] = {h.nb, h.nbr, h.nbase, h.coef, h.cw, h.m6, h.enb, h.ecf, h.ud, h.vflags, h.vparams, h.stim, h.u, h.h0, h.h1, h.x, h.b, h.V,
                    h.hist_u, h.hist_h, h.lat, h.part, h.sync, h.st, h.prof};
    for (void* p : ptrs) dev_free(p, 0);
    h = InstHost();
}

}  // namespace

struct phs_engine {
    int prec = PHS_PREC_F32;
    int device = 0;
    int sms = 0;
    std::vector<InstHost> inst;
    unsigned int* abort_word = nullptr;
    void* d_desc = nullptr;
    size_t d_desc_bytes = 0;
    int4* d_map = nullptr;
    size_t d_map_n = 0;
    long long launches = 0;
    bool broken = false;
    // cached launch plan (rebuilt when the instance set changes)
    bool dirty = true;
    std::vector<int> act;
    std::vector<std::pair<size_t, int>> waves;
    int plan_cps = -1;
    bool plan_edge = false;  // the plan launches the edge-term kernel
    bool auto_balance = true;  // rebalance on the 2nd and 3rd advance after the instance set changes
    int auto_left = 0;
    long long auto_mark = 0;   // launch count when the set changed / at the last automatic rebalance
    bool auto_prof = false;    // the phase timers were switched on by the automatic balancing
    // CUDA graphs of the launch sequence, keyed by steps per launch
    std::map<long long, cudaGraphExec_t> graphs;
    bool graphs_ok = true;
    int variant = -1;        // step-kernel variant (-1: default of the precision)
    bool profile = false;    // per-instance phase timers
    bool test_overcount = false;  // test hook: first team waits for one CTA too many
    int default_cps = 0;     // CTAs per SM when advance() is given 0 (0: occupancy limit)
    int wave_instances = 0;  // instances per launch wave (0: as many as the grid holds)
    bool compact_nb = true;  // instances read the compact neighbour table when they have one
};

namespace {

template <typename T>
int occupancy_for(int* ctas, int variant, bool edge = false) {
    const void* fn = step_fn<T>(variant, edge);
    const int smem = dyn_smem_of((int)sizeof(T), variant);
    if (smem > 0) {
        cudaError_t a = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (a != cudaSuccess) { set_last_error("ring shared memory", a); return PHS_ERR_CUDA; }
    }
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, fn, threads_of((int)sizeof(T), variant), smem);
    if (e != cudaSuccess) { set_last_error("occupancy", e); return PHS_ERR_CUDA; }
    return PHS_OK;
}

template <typename T>
void fill_dev(T* p, long long n, T v, cudaStream_t s) {
    if (n <= 0) return;
    long long blocks = std::min<long long>((n + 255) / 256, 65535);
    fill_kernel<T><<<(unsigned)blocks, 256, 0, s>>>(p, n, v);
}

// Device-side form of validate_desc's table checks (device_tables instances).
template <typename T>
__global__ void check_tables(long long n, const int32_t* nb, const T* coef, const T* cw, const uint8_t* m6,
                             const int32_t* enb, const T* ecf, unsigned int* err) {
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n; r += (long long)gridDim.x * blockDim.x) {
        bool bad = false;
        for (int k = 0; k < 6; ++k) {
            const int32_t q = nb[6 * r + k];
            bad |= (q < 0 || q >= n);
            if (coef) bad |= !isfinite((double)coef[6 * r + k]);
        }
        if (cw) bad |= !isfinite((double)cw[r]) || (m6[r] & 0xC0u);
        if (enb) {
            for (int k = 0; k < 12; ++k) bad |= (enb[12 * r + k] < 0 || enb[12 * r + k] >= n);
            for (int k = 0; k < 6; ++k) bad |= !isfinite((double)ecf[6 * r + k]);
        }
        if (bad) atomicOr(err, 1u);
    }
}

// ---- compact neighbour table (decode_nb)
// Whether slot k of row v has a neighbour the operator reads: its coefficient
// is nonzero, the test tile_lap makes.
template <typename T>
__device__ __forceinline__ bool nb_present(const T* coef, const T* cw, const uint8_t* m6, long long v, int k) {
    if (cw) return ((m6[v] >> k) & 1u) && cw[v] != T(0);
    return coef[6 * v + k] != T(0);
}

// flags[k] bit 0: some present neighbour of slot k is not n + 1; bit 1: not n - 1.
template <typename T>
__global__ void nb_slot_kinds(long long n, const int32_t* nb, const T* coef, const T* cw, const uint8_t* m6,
                              unsigned int* flags) {
    unsigned int f[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        for (int k = 0; k < 6; ++k) {
            if (!nb_present(coef, cw, m6, v, k)) continue;
            const long long dq = (long long)nb[6 * v + k] - v;
            f[k] |= (dq != 1 ? 1u : 0u) | (dq != -1 ? 2u : 0u);
        }
    }
    for (int k = 0; k < 6; ++k) {
        unsigned int a = f[k];
        for (int o = 16; o > 0; o >>= 1) a |= __shfl_xor_sync(0xffffffffu, a, o);
        if ((threadIdx.x & 31) == 0 && a) atomicOr(flags + k, a);
    }
}

// Largest over the rows of (diagonal of -L) + (sum of its off-diagonal
// magnitudes), the upper bound Gershgorin's theorem gives for the eigenvalues of -L;
// rounded up to FP32, whose bit patterns of non-negative values order as
// integers (NaN above all).
template <typename T>
__global__ void row_bound(long long n, const T* coef, const T* cw, const uint8_t* m6, const T* ecf, unsigned int* out) {
    float b = 0.f;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        double diag = 0.0, off = 0.0;
        for (int k = 0; k < 6; ++k) {
            const double c = cw ? (((m6[v] >> k) & 1u) ? (double)cw[v] : 0.0) : (double)coef[6 * v + k];
            diag += c;
            off += fabs(c);
            if (ecf) off += 2.0 * fabs((double)ecf[6 * v + k]);
        }
        const float r = __double2float_ru(diag + off);
        if (!(r <= b)) b = r;
    }
    if (!(b >= 0.f)) b = __int_as_float(0x7fffffff);
    unsigned int u = __float_as_uint(b);
    for (int o = 16; o > 0; o >>= 1) u = max(u, __shfl_xor_sync(0xffffffffu, u, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, u);
}

// One CTA of 256 threads per 512-voxel block: for slots 2..5 the base offset
// (middle of the block's range over present neighbours) and the int16
// residuals; *fail set when a block's range does not fit.  Voxels past n
// (padding) get zeros.
template <typename T>
__global__ void nb_compact(long long n, const int32_t* nb, const T* coef, const T* cw, const uint8_t* m6,
                           int16_t* nbr, int32_t* nbase, unsigned int* fail) {
    __shared__ long long lo[8][4], hi[8][4];
    __shared__ int32_t base[4];
    const long long v0 = (long long)blockIdx.x * 512;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long mn[4], mx[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) { mn[r] = LLONG_MAX; mx[r] = LLONG_MIN; }
    for (int h = 0; h < 2; ++h) {
        const long long v = v0 + h * 256 + threadIdx.x;
        if (v >= n) continue;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (!nb_present(coef, cw, m6, v, r + 2)) continue;
            const long long dq = (long long)nb[6 * v + r + 2] - v;
            mn[r] = min(mn[r], dq);
            mx[r] = max(mx[r], dq);
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[r] = min(mn[r], (long long)__shfl_xor_sync(0xffffffffu, mn[r], o));
            mx[r] = max(mx[r], (long long)__shfl_xor_sync(0xffffffffu, mx[r], o));
        }
        if (lane == 0) { lo[w][r] = mn[r]; hi[w][r] = mx[r]; }
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        const int r = threadIdx.x;
        long long a = LLONG_MAX, b = LLONG_MIN;
        for (int q = 0; q < 8; ++q) { a = min(a, lo[q][r]); b = max(b, hi[q][r]); }
        long long bs = 0;
        if (a <= b) {
            bs = a + (b - a) / 2;
            if (b - bs > 32767 || a - bs < -32768 || bs > INT_MAX / 2 || bs < INT_MIN / 2) atomicOr(fail, 1u);
        }
        base[r] = (int32_t)bs;
        nbase[blockIdx.x * 4 + r] = (int32_t)bs;
    }
    __syncthreads();
    for (int h = 0; h < 2; ++h) {
        const long long v = v0 + h * 256 + threadIdx.x;
        long long d[4] = {0, 0, 0, 0};
        if (v < n) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (nb_present(coef, cw, m6, v, r + 2)) d[r] = (long long)nb[6 * v + r + 2] - v - base[r];
        }
        short res[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) res[r] = (short)max(-32768ll, min(32767ll, d[r]));
        reinterpret_cast<short4*>(nbr)[v] = make_short4(res[0], res[1], res[2], res[3]);
    }
}

// Copy n doubles (host, or device when on_device) into a new array of T of
// alloc_n >= n elements (the tail is zero).
template <typename T>
int upload_converted(void** dst, const double* src, long long n, bool on_device, long long alloc_n) {
    PHS_CUDA_TRY(dev_alloc(dst, (size_t)alloc_n * sizeof(T), 0));
    if (alloc_n > n) PHS_CUDA_TRY(cudaMemset((char*)*dst + (size_t)n * sizeof(T), 0, (size_t)(alloc_n - n) * sizeof(T)));
    if (sizeof(T) == 8) {
        PHS_CUDA_TRY(cudaMemcpy(*dst, src, (size_t)n * 8, cudaMemcpyDefault));
        return PHS_OK;
    }
    double* tmp = nullptr;
    cudaError_t e = cudaSuccess;
    if (!on_device) {
        PHS_CUDA_TRY(dev_alloc((void**)&tmp, (size_t)n * 8, 0));
        e = cudaMemcpy(tmp, src, (size_t)n * 8, cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) {
        long long blocks = std::min<long long>((n + 255) / 256, 65535);
        convert_kernel<T><<<(unsigned)std::max<long long>(blocks, 1), 256>>>(on_device ? src : tmp, (T*)*dst, n);
        e = cudaDeviceSynchronize();
    }
    dev_free(tmp, 0);
    if (e != cudaSuccess) { set_last_error("upload_converted", e); return PHS_ERR_CUDA; }
    return PHS_OK;
}

int validate_desc(const phs_instance_desc* d) {
    if (!d || d->n_voxel <= 0 || d->n_voxel > (1ll << 31) - 1) return PHS_ERR_BAD_ARG;
    if (d->model != PHS_MODEL_MS && d->model != PHS_MODEL_AP) return PHS_ERR_BAD_ARG;
    if (d->restart < 1 || d->restart > kMaxRestart) return PHS_ERR_BAD_ARG;
    if (!d->nb6 || !d->vflags) return PHS_ERR_BAD_ARG;
    if (!d->coef6 && !(d->cw && d->mask6)) return PHS_ERR_BAD_ARG;
    if (d->n_steps < 0 || (d->n_steps > 0 && !d->stim)) return PHS_ERR_BAD_ARG;
    if (d->n_samples < 0 || d->sample_stride < 0 || d->maxiter < 1) return PHS_ERR_BAD_ARG;
    if (!(d->dt > 0.0)) return PHS_ERR_BAD_ARG;
    if ((d->nb_edge == nullptr) != (d->coef_edge == nullptr)) return PHS_ERR_BAD_ARG;
    if (d->device_tables) return PHS_OK;   // checked on the device after the copy (check_tables)
    const long long n = d->n_voxel;
    for (long long i = 0; i < 6 * n; ++i) {
        int32_t q = d->nb6[i];
        if (q < 0 || q >= n) return PHS_ERR_BAD_TABLE;
        if (d->coef6 && !std::isfinite(d->coef6[i])) return PHS_ERR_BAD_TABLE;
    }
    if (d->cw)
        for (long long i = 0; i < n; ++i)
            if (!std::isfinite(d->cw[i]) || (d->mask6[i] & 0xC0u)) return PHS_ERR_BAD_TABLE;
    if (d->nb_edge) {
        for (long long i = 0; i < 12 * n; ++i)
            if (d->nb_edge[i] < 0 || d->nb_edge[i] >= n) return PHS_ERR_BAD_TABLE;
        for (long long i = 0; i < 6 * n; ++i)
            if (!std::isfinite(d->coef_edge[i])) return PHS_ERR_BAD_TABLE;
    }
    return PHS_OK;
}

// Build the compact neighbour table (decode_nb) and the eigenvalue bound of an
// instance whose tables are on the device (h.nb with the coefficients).  Leaves h.nbr null when a
// present neighbour of slot 0 is not n + 1, one of slot 1 not n - 1, or a
// block's offsets of another slot do not fit int16.
template <typename T>
int build_compact_nb(InstHost& h) {
    const long long n = h.n;
    unsigned int* d_w = nullptr;
    PHS_CUDA_TRY(dev_alloc((void**)&d_w, 8 * sizeof(unsigned int), 0));
    unsigned int w[8] = {};
    cudaError_t ce = cudaMemset(d_w, 0, 8 * sizeof(unsigned int));
    const long long blocks = std::max<long long>(1, std::min<long long>((n + 255) / 256, 4096));
    if (ce == cudaSuccess) {
        nb_slot_kinds<T><<<(unsigned)blocks, 256>>>(n, (const int32_t*)h.nb, (const T*)h.coef, (const T*)h.cw,
                                                    (const uint8_t*)h.m6, d_w);
        row_bound<T><<<(unsigned)blocks, 256>>>(n, (const T*)h.coef, (const T*)h.cw, (const uint8_t*)h.m6,
                                                (const T*)h.ecf, d_w + 7);
        ce = cudaGetLastError();
    }
    if (ce == cudaSuccess) ce = cudaMemcpy(w, d_w, 8 * sizeof(unsigned int), cudaMemcpyDeviceToHost);
    float bound = 0.f;
    memcpy(&bound, &w[7], sizeof(bound));
    h.bound = (double)bound;
    if (ce == cudaSuccess && !(w[0] & 1u) && !(w[1] & 2u)) {
        const long long nblk = h.ldv / 512;
        ce = dev_alloc((void**)&h.nbr, (size_t)h.ldv * 4 * sizeof(int16_t), 0);
        if (ce == cudaSuccess) ce = dev_alloc((void**)&h.nbase, (size_t)nblk * 4 * sizeof(int32_t), 0);
        if (ce == cudaSuccess) ce = cudaMemset(d_w + 6, 0, sizeof(unsigned int));
        if (ce == cudaSuccess) {
            nb_compact<T><<<(unsigned)nblk, 256>>>(n, (const int32_t*)h.nb, (const T*)h.coef, (const T*)h.cw,
                                                   (const uint8_t*)h.m6, h.nbr, h.nbase, d_w + 6);
            ce = cudaGetLastError();
        }
        if (ce == cudaSuccess) ce = cudaMemcpy(w + 6, d_w + 6, sizeof(unsigned int), cudaMemcpyDeviceToHost);
        if (ce != cudaSuccess || w[6] != 0u) {
            dev_free(h.nbr, 0);
            dev_free(h.nbase, 0);
            h.nbr = nullptr;
            h.nbase = nullptr;
        }
    }
    dev_free(d_w, 0);
    if (ce != cudaSuccess) { set_last_error("build_compact_nb", ce); return PHS_ERR_CUDA; }
    return PHS_OK;
}

template <typename T>
int add_instance(phs_engine* e, const phs_instance_desc* d, int* slot) {
    int rc = validate_desc(d);
    if (rc != PHS_OK) return rc;
    InstHost h;
    h.used = true;
    h.d = *d;
    h.n = d->n_voxel;
    const int vpt = sizeof(T) == 8 ? kVptF64 : kVptF32Min;   // allocations cover every variant's tiles
    const long long tile = (long long)kThreads * vpt;
    h.n_tiles = (int)((h.n + tile - 1) / tile);
    h.m = (int)std::min<long long>(d->restart, h.n);
    const size_t n = (size_t)h.n;
    // per-voxel arrays hold a whole number of the largest tile (zero tail), so
    // a tile's slice of any of them can be copied whole
    const size_t np = (n + kPadVoxels - 1) / kPadVoxels * kPadVoxels;
    h.ldv = (long long)np;
    auto fail = [&](int code) {
        free_inst(h);
        cudaStreamSynchronize(0);
        return code;
    };
#define PHS_ALLOC(ptr, bytes)                                            \
    do {                                                                 \
        cudaError_t _e = dev_alloc((void**)&(ptr), (bytes), 0);          \
        if (_e != cudaSuccess) { set_last_error("dev_alloc", _e); return fail(PHS_ERR_OOM); } \
    } while (0)
    // tables: host arrays, or device arrays when device_tables (cudaMemcpyDefault)
    const bool dev = d->device_tables != 0;
    auto copy_in = [&](void* dst, const void* src, size_t bytes, size_t alloc_bytes) {
        if (alloc_bytes > bytes && cudaMemset((char*)dst + bytes, 0, alloc_bytes - bytes) != cudaSuccess) return false;
        return cudaMemcpy(dst, src, bytes, cudaMemcpyDefault) == cudaSuccess;
    };
    PHS_ALLOC(h.nb, np * 6 * sizeof(int32_t));
    if (!copy_in(h.nb, d->nb6, n * 6 * sizeof(int32_t), np * 6 * sizeof(int32_t))) return fail(PHS_ERR_CUDA);
    if (d->cw) {
        if ((rc = upload_converted<T>(&h.cw, d->cw, (long long)n, dev, (long long)np)) != PHS_OK) return fail(rc);
        PHS_ALLOC(h.m6, np);
        if (!copy_in(h.m6, d->mask6, n, np)) return fail(PHS_ERR_CUDA);
    } else {
        if ((rc = upload_converted<T>(&h.coef, d->coef6, (long long)n * 6, dev, (long long)np * 6)) != PHS_OK)
            return fail(rc);
    }
    if (d->nb_edge) {
        PHS_ALLOC(h.enb, np * 12 * sizeof(int32_t));
        if (!copy_in(h.enb, d->nb_edge, n * 12 * sizeof(int32_t), np * 12 * sizeof(int32_t))) return fail(PHS_ERR_CUDA);
        if ((rc = upload_converted<T>(&h.ecf, d->coef_edge, (long long)n * 6, dev, (long long)np * 6)) != PHS_OK)
            return fail(rc);
    }
    PHS_ALLOC(h.vflags, np);
    if (!copy_in(h.vflags, d->vflags, n, np)) return fail(PHS_ERR_CUDA);
    if (d->vparams) {
        if ((rc = upload_converted<T>(&h.vparams, d->vparams, (long long)n * 5, dev, (long long)np * 5)) != PHS_OK)
            return fail(rc);
    }
    if (dev) {
        // the checks validate_desc makes on host tables, on the copies
        unsigned int* d_err = nullptr;
        if (dev_alloc((void**)&d_err, sizeof(unsigned int), 0) != cudaSuccess) return fail(PHS_ERR_OOM);
        unsigned int h_err = 0;
        cudaError_t ce = cudaMemset(d_err, 0, sizeof(unsigned int));
        if (ce == cudaSuccess) {
            const long long blocks = std::max<long long>(1, std::min<long long>(((long long)n + 255) / 256, 65535));
            check_tables<T><<<(unsigned)blocks, 256>>>((long long)n, (const int32_t*)h.nb, (const T*)h.coef,
                                                       (const T*)h.cw, (const uint8_t*)h.m6, (const int32_t*)h.enb,
                                                       (const T*)h.ecf, d_err);
            ce = cudaGetLastError();
        }
        if (ce == cudaSuccess) ce = cudaMemcpy(&h_err, d_err, sizeof(h_err), cudaMemcpyDeviceToHost);
        dev_free(d_err, 0);
        if (ce != cudaSuccess) { set_last_error("check_tables", ce); return fail(PHS_ERR_CUDA); }
        if (h_err) return fail(PHS_ERR_BAD_TABLE);
    }
    if ((rc = build_compact_nb<T>(h)) != PHS_OK) return fail(rc);
    const size_t ns = (size_t)std::max<int64_t>(d->n_steps, 1);
    PHS_ALLOC(h.stim, ns);
    if (d->n_steps > 0) {
        if (cudaMemcpy(h.stim, d->stim, (size_t)d->n_steps, cudaMemcpyHostToDevice) != cudaSuccess) return fail(PHS_ERR_CUDA);
    } else {
        cudaMemset(h.stim, 0, ns);
    }
    PHS_ALLOC(h.u, np * sizeof(T));
    PHS_ALLOC(h.h0, np * sizeof(T));
    PHS_ALLOC(h.h1, np * sizeof(T));
    PHS_ALLOC(h.x, np * sizeof(T));
    PHS_ALLOC(h.b, np * sizeof(T));
    PHS_ALLOC(h.V, np * (size_t)(h.m + 1) * sizeof(T));
    PHS_ALLOC(h.ud, np * 2 * sizeof(T));
    const size_t S = (size_t)std::max(d->n_samples, 1);
    PHS_ALLOC(h.hist_u, S * n * sizeof(T));
    if (d->save_h) PHS_ALLOC(h.hist_h, S * n * sizeof(T));
    PHS_ALLOC(h.lat, np * sizeof(int32_t));
    h.part_half = (long long)groups_of<T>(h.n_tiles) * (h.m + 2);
    PHS_ALLOC(h.part, (size_t)h.part_half * 2 * sizeof(double));
    PHS_ALLOC(h.sync, sizeof(TeamSync));
    PHS_ALLOC(h.st, sizeof(InstState));
#undef PHS_ALLOC
    fill_dev<T>((T*)h.u, (long long)np, (T)d->u0, 0);
    fill_dev<T>((T*)h.h0, (long long)np, (T)d->h0, 0);
    fill_dev<T>((T*)h.h1, (long long)np, (T)d->h0, 0);
    fill_dev<T>((T*)h.x, (long long)np, (T)0, 0);
    fill_dev<T>((T*)h.b, (long long)np, (T)0, 0);
    cudaMemset(h.V, 0, np * (size_t)(h.m + 1) * sizeof(T));
    cudaMemset(h.ud, 0, np * 2 * sizeof(T));
    cudaMemset(h.hist_u, 0, S * n * sizeof(T));
    if (h.hist_h) cudaMemset(h.hist_h, 0, S * n * sizeof(T));
    cudaMemset(h.lat, 0xff, np * sizeof(int32_t));
    cudaMemset(h.part, 0, (size_t)h.part_half * 2 * sizeof(double));
    cudaMemset(h.sync, 0, sizeof(TeamSync));
    InstState st{};
    st.step = 0;
    st.id_save = 0;
    st.pending = -1;
    st.status = PHS_OK;
    st.hbuf = 0;
    cudaMemcpy(h.st, &st, sizeof(st), cudaMemcpyHostToDevice);
    cudaError_t ce = cudaDeviceSynchronize();
    if (ce != cudaSuccess) { set_last_error("add_instance", ce); return fail(PHS_ERR_CUDA); }
    h.st_host = st;
    h.finished = (d->n_steps == 0);
    // find a free slot
    int s = -1;
    for (size_t i = 0; i < e->inst.size(); ++i)
        if (!e->inst[i].used) { s = (int)i; break; }
    if (s < 0) { s = (int)e->inst.size(); e->inst.push_back(InstHost()); }
    if (e->profile) {
        if (dev_alloc((void**)&h.prof, kProfSlots * sizeof(unsigned long long), 0) == cudaSuccess)
            cudaMemset(h.prof, 0, kProfSlots * sizeof(unsigned long long));
    }
    // columns per step until they are known.  A guess for the team sizes of the first
    // launch only, through the two stiffnesses at hand (Mitchell-Schaeffer shells, hg
    // 0.94: 4.7, Aliev-Panfilov, hg 0.6: 1.8; 24 and 19 in full cycles): at another
    // lattice constant or step it may be off by a factor, and the measured costs
    // take its place at the first rebalancing
    const double hg = std::min(1.0, 0.25 * d->dt * h.bound);
    h.kavg = d->full_cycles ? 10.0 + 15.0 * hg : 1.0 + 4.4 * hg * hg * hg;
    e->inst[s] = h;
    pool_update(0);
    e->dirty = true;
    e->auto_left = 2;
    e->auto_mark = e->launches;
    *slot = s;
    return PHS_OK;
}

// Which solves use the Chebyshev basis.  hg: the half width of the interval
// of A - I.  Its Gram matrix stays positive definite in FP64 longer than a solve
// needs where it converges by 4 and more per column; on the stiff side it is lost
// after 22-30 columns (hg 3 and 15, discs and rough residuals) or, for plane
// fronts, after 10-17 (FP32 from hg 5, FP64 from hg 3 on at tol 1e-9).  Early
// exit: with restarts of up to 20 columns a lost matrix costs little, the cycle
// ends in a true residual and the solve goes on (64 x 64 sheet, plane front, more
// columns than Arnoldi's, FP32 at tol 1e-6 / FP64 at 1e-9: 1 / 30 % at hg 3, 6 / 13 %
// at 5, 21 / 12 % at 15, 17 / 17 % at 60, at half the passes per column).  Full cycles want rounding level: up to
// hg 1.25 (Mitchell-Schaeffer at 0.05 ms and 0.4 mm: 0.94) that takes 21-28
// columns; beyond, Arnoldi.
bool cheb_rule(bool full_cycles, int m, double hg) {
    if (!(hg >= 0.0) || !std::isfinite(hg)) return false;
    return hg <= 1.25 || (!full_cycles && m <= 20);
}

template <typename T>
InstDev<T> make_dev(const InstHost& h, int vpt, bool compact_nb) {
    InstDev<T> I{};
    I.nb = (const int32_t*)h.nb;
    if (compact_nb && h.nbr) {
        I.nbr = h.nbr;
        I.nbase = h.nbase;
    }
    I.coef = (const T*)h.coef;
    I.cw = (const T*)h.cw;
    I.m6 = (const uint8_t*)h.m6;
    I.enb = (const int32_t*)h.enb;
    I.ecf = (const T*)h.ecf;
    I.vflags = (const uint8_t*)h.vflags;
    I.vparams = (const T*)h.vparams;
    I.stim = (const uint8_t*)h.stim;
    I.u = (T*)h.u;
    I.h0 = (T*)h.h0;
    I.h1 = (T*)h.h1;
    I.x = (T*)h.x;
    I.b = (T*)h.b;
    I.V = (T*)h.V;
    I.ldv = h.ldv;
    I.ud = (T*)h.ud;
    I.guess = h.d.guess;
    I.hist_u = (T*)h.hist_u;
    I.hist_h = (T*)h.hist_h;
    I.lat = h.lat;
    I.part = h.part;
    I.part_half = h.part_half;
    I.sync = h.sync;
    I.st = h.st;
    I.prof = h.prof;
    T raw[5];
    for (int q = 0; q < 5; ++q) raw[q] = (T)h.d.params[q];
    model_form<T>(h.d.model, raw, I.params);
    I.dt = (T)h.d.dt;
    I.half_dt = (T)h.d.dt / T(2);
    I.jmag = (T)h.d.j_stim;
    I.tol = h.d.tol;
    I.atol = h.d.atol;
    I.n = h.n;
    I.n_steps = h.d.n_steps;
    I.tb_steps = h.d.tblock_steps;
    I.n_tiles = tiles_of(h.n, vpt);
    I.gt = group_tiles<T>(I.n_tiles);
    I.n_groups = groups_of<T>(I.n_tiles);
    I.model = h.d.model;
    I.m = h.m;
    I.maxiter = h.d.maxiter;
    I.full_cycles = h.d.full_cycles;
    I.stride = h.d.sample_stride;
    I.n_samples = h.d.n_samples;
    I.save_h = h.d.save_h;
    // Isotropic rows: A = I - dt/2 L has its eigenvalues in 1 + [0, 2 hg] (its rows are
    // those of a symmetric matrix scaled by c_n >= 0).  With cross terms the
    // off-diagonal magnitudes exceed the diagonal and the rows are not symmetric, so
    // eigenvalues below 1 or off the real axis are not excluded: the interval is a
    // heuristic there, the columns may grow outside it, and the test for a lost Gram
    // matrix is what guards the solve (fibre shells: column counts are Arnoldi's)
    const double hg = 0.5 * (0.5 * h.d.dt) * h.bound;
    const double delta = std::max(hg, 1.0 / 16), theta = 1.0 + hg;
    I.cheb = cheb_rule(h.d.full_cycles != 0, h.m, hg) ? 1 : 0;
    I.cheb_a = (T)((1.0 - theta) / delta);
    I.cheb_b = (T)(-0.5 * h.d.dt / delta);
    // the centre and width that the stored constants stand for
    I.delta = -(double)I.half_dt / (double)I.cheb_b;
    I.theta = 1.0 - I.delta * (double)I.cheb_a;
    I.inv_delta = 1.0 / I.delta;
    I.t1 = -I.theta / I.delta;
    return I;
}

// Split G CTAs over the instances.  A team of P CTAs over `tiles` tiles takes
// time proportional to (cost per tile) x ceil(tiles / P): its CTAs walk their
// tiles one after another and the one with the most tiles sets the pace.  The
// cost of an instance is `weight` (voxels times the cost of a step in units of
// one column, or the measured CTA-time per step), per tile weight /
// tiles.  Starting from one CTA each, the instance with the longest time
// receives the fewest CTAs that lower its tiles-per-CTA count, until the CTAs
// run out or the longest one cannot be helped; CTAs left over (when every team
// already has one CTA per tile, or the longest would need more than remain) go
// to no one.  Never more CTAs than tiles.
// A step costs as much as this many columns beside its columns (right-hand side,
// update, reaction: 12 against 5.3 CTA-ns per voxel in a batch of 24 shells, for
// both models).
constexpr double kStepCost = 2.3;
std::vector<int> team_sizes(const std::vector<int>& tiles, const std::vector<double>& weight, int G) {
    const int A = (int)tiles.size();
    std::vector<int> P(A, 1);
    int used = A;
    auto per_tile = [&](int i) { return weight[i] / std::max(tiles[i], 1); };
    auto span = [&](int i, int p) { return (tiles[i] + p - 1) / p; };
    while (used < G) {
        int worst = -1;
        double wt = -1.0;
        for (int i = 0; i < A; ++i) {
            const double t = per_tile(i) * span(i, P[i]);
            if (t > wt) { wt = t; worst = i; }
        }
        if (worst < 0) break;
        const int cur = span(worst, P[worst]);
        if (cur <= 1) break;                                   // one tile per CTA already
        const int need = (tiles[worst] + (cur - 1) - 1) / (cur - 1);   // fewest CTAs with span cur - 1
        if (used + (need - P[worst]) > G) break;
        used += need - P[worst];
        P[worst] = need;
    }
    return P;
}

// The variant a launch uses: the configured one, or its int32-table twin when
// it reads compact tables and an unfinished instance has none (or the engine's
// compact tables are off).
template <typename T>
int variant_of(const phs_engine* e) {
    int v = e->variant >= 0 ? e->variant : (sizeof(T) == 8 ? kDefaultF64 : kDefaultF32);
    if (sizeof(T) == 4 && kTwinF32[v] >= 0) {
        bool all = e->compact_nb;
        for (const auto& h : e->inst)
            if (h.used && !h.finished && !h.nbr) all = false;
        if (!all) v = kTwinF32[v];
    }
    return v;
}

void drop_graphs(phs_engine* e) {
    for (auto& kv : e->graphs) cudaGraphExecDestroy(kv.second);
    e->graphs.clear();
}

template <typename T>
cudaError_t launch_waves(phs_engine* e, long long n_steps, cudaStream_t stream) {
    for (auto& wv : e->waves) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)wv.second);
        const int variant = variant_of<T>(e);
        cfg.blockDim = dim3((unsigned)threads_of((int)sizeof(T), variant));
        cfg.dynamicSmemBytes = (size_t)dyn_smem_of((int)sizeof(T), variant);
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const InstDev<T>* dd = (const InstDev<T>*)e->d_desc;
        const int4* mp = e->d_map + wv.first;
        long long ns = n_steps;
        unsigned int* ab = e->abort_word;
        void* args[] = {(void*)&dd, (void*)&mp, (void*)&ns, (void*)&ab};
        cudaError_t ce = cudaLaunchKernelExC(&cfg, step_fn<T>(variant, e->plan_edge), args);
        if (ce != cudaSuccess) return ce;
    }
    return cudaSuccess;
}

// Whether a wave's passes prefetch their next tiles into L2: when what a step
// streams is over twice L2.  With all loads of a tile in flight
// together the prefetch only helps where those go to DRAM, and costs issue slots
// elsewhere.  Shells of 50k-400k voxels, ms per step with and without: 16 (2.2M
// voxels, 160 MB) 0.144 / 0.131, 24 (3.9M) 0.255 / 0.248, 32 (5.2M, 380 MB)
// 0.317 / 0.327, 64 (10.9M) 0.652 / 0.729.
template <typename T>
bool plan_prefetch(const phs_engine* e, const std::vector<int>& act, size_t w0, size_t w1) {
    int l2 = 0;
    if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, e->device) != cudaSuccess || l2 <= 0) return false;
    double bytes = 0.0;
    for (size_t i = w0; i < w1; ++i) {
        const InstHost& h = e->inst[act[i]];
        const double tables = (h.nbr ? 8 : 24) + (h.cw ? sizeof(T) + 1 : 6 * sizeof(T)) + (h.enb ? 48 + 6 * sizeof(T) : 0) + 1;
        bytes += (double)h.n * (tables + sizeof(T) * (6.0 + h.kavg) + 4.0);
    }
    return bytes > 2.0 * l2;
}

// (Re)build the launch plan: device descriptors, team map and waves.
template <typename T>
int build_plan(phs_engine* e, int cps, bool edge) {
    // earlier launches may still read the old descriptors
    PHS_CUDA_TRY(cudaDeviceSynchronize());
    const int G = e->sms * cps;
    std::vector<int> act;
    for (size_t i = 0; i < e->inst.size(); ++i)
        if (e->inst[i].used && !e->inst[i].finished) act.push_back((int)i);
    e->act = act;
    e->waves.clear();
    drop_graphs(e);
    e->plan_cps = cps;
    e->plan_edge = edge;
    e->dirty = false;
    if (act.empty()) return PHS_OK;
    std::vector<InstDev<T>> descs;
    descs.reserve(act.size());
    const int vpt = vpt_of((int)sizeof(T), variant_of<T>(e));
    for (int i : act) descs.push_back(make_dev<T>(e->inst[i], vpt, e->compact_nb));
    size_t bytes = descs.size() * sizeof(InstDev<T>);
    if (bytes > e->d_desc_bytes) {
        dev_free(e->d_desc, 0);
        e->d_desc = nullptr;
        e->d_desc_bytes = 0;
        PHS_CUDA_TRY(dev_alloc(&e->d_desc, bytes, 0));
        e->d_desc_bytes = bytes;
    }
    PHS_CUDA_TRY(cudaMemcpy(e->d_desc, descs.data(), bytes, cudaMemcpyHostToDevice));

    // waves of at most G instances (fewer with wave_instances: each wave is a
    // launch of its own over the whole grid, so the instances of a wave share
    // the L2 with fewer others)
    std::vector<int4> map_all;
    std::vector<std::pair<size_t, int>>& waves = e->waves;  // (offset into map, grid)
    const size_t per_wave = (size_t)((e->wave_instances > 0) ? std::min(G, e->wave_instances) : G);
    for (size_t w0 = 0; w0 < act.size(); w0 += per_wave) {
        size_t w1 = std::min(act.size(), w0 + per_wave);
        std::vector<int> tiles;
        std::vector<double> weight;
        bool measured = true;
        for (size_t i = w0; i < w1; ++i) measured = measured && e->inst[act[i]].weight > 0.0;
        for (size_t i = w0; i < w1; ++i) {
            const InstHost& h = e->inst[act[i]];
            tiles.push_back(groups_of<T>(tiles_of(h.n, vpt)));
            weight.push_back(measured ? h.weight : (double)h.n * (kStepCost + h.kavg));
        }
        std::vector<int> P = team_sizes(tiles, weight, G);
        for (size_t i = w0; i < w1; ++i) e->inst[act[i]].team = P[i - w0];
        const int prefetch = plan_prefetch<T>(e, act, w0, w1) ? 1 : 0;
        size_t off = map_all.size();
        int grid = 0;
        for (size_t i = w0; i < w1; ++i) {
            int p = P[i - w0];
            // test hook: the first team expects one CTA that is never launched, so
            // its first barrier can only end through the bounded wait
            const int claimed = p + ((e->test_overcount && i == w0) ? 1 : 0);
            for (int r = 0; r < p; ++r) map_all.push_back(make_int4((int)i, r, claimed, prefetch));
            grid += p;
        }
        waves.push_back({off, grid});
    }
    if (map_all.size() > e->d_map_n) {
        dev_free(e->d_map, 0);
        e->d_map = nullptr;
        e->d_map_n = 0;
        PHS_CUDA_TRY(dev_alloc((void**)&e->d_map, map_all.size() * sizeof(int4), 0));
        e->d_map_n = map_all.size();
    }
    PHS_CUDA_TRY(cudaMemcpy(e->d_map, map_all.data(), map_all.size() * sizeof(int4), cudaMemcpyHostToDevice));
    // The launch may be on a stream that does not wait for the legacy one (any
    // non-blocking stream), on which the two arrays were allocated and filled, and
    // a copy from pageable memory may return before its transfer has landed.
    PHS_CUDA_TRY(cudaStreamSynchronize(0));
    return PHS_OK;
}

template <typename T>
int advance_impl(phs_engine* e, long long n_steps, int ctas_per_sm, cudaStream_t stream, bool sync) {
    if (e->broken) return PHS_ERR_STATE;
    if (n_steps <= 0) return PHS_OK;
    // automatic balancing: the launch after an instance set change runs with the
    // phase timers on (unless the caller has them on already), the next two
    // re-split the CTAs by the measured cost, then the timers go off again
    if (e->auto_balance && e->auto_left > 0 && !e->profile) {
        const int rp = phs_engine_config(e, PHS_CFG_PROFILE, 1);
        if (rp != PHS_OK) return rp;
        e->auto_prof = true;
    }
    if (e->auto_balance && e->auto_left > 0 && e->launches > e->auto_mark) {
        const int rb = phs_engine_rebalance(e);
        if (rb != PHS_OK) return rb;
        e->auto_left -= 1;
        e->auto_mark = e->launches;
        if (e->auto_left == 0 && e->auto_prof) {
            const int rp = phs_engine_config(e, PHS_CFG_PROFILE, 0);
            if (rp != PHS_OK) return rp;
            e->auto_prof = false;
        }
    }
    // the edge-term kernel only when an unfinished instance is anisotropic
    bool edge = false;
    for (const auto& h : e->inst)
        if (h.used && !h.finished && h.enb) edge = true;
    int occ = 0;
    int rc = occupancy_for<T>(&occ, variant_of<T>(e), edge);
    if (rc != PHS_OK) return rc;
    if (occ < 1) return PHS_ERR_CUDA;
    if (ctas_per_sm <= 0) ctas_per_sm = e->default_cps;
    int cps = (ctas_per_sm > 0) ? std::min(ctas_per_sm, occ) : occ;
    if (e->dirty || cps != e->plan_cps || edge != e->plan_edge) {
        rc = build_plan<T>(e, cps, edge);
        if (rc != PHS_OK) return rc;
    }
    const std::vector<int>& act = e->act;
    if (act.empty()) return PHS_OK;
    cudaError_t ce = cudaSuccess;
    bool launched = false;
    if (stream != nullptr && e->graphs_ok) {
        auto it = e->graphs.find(n_steps);
        if (it == e->graphs.end()) {
            cudaGraph_t g = nullptr;
            cudaGraphExec_t ge = nullptr;
            ce = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal);
            if (ce == cudaSuccess) {
                cudaError_t le = launch_waves<T>(e, n_steps, stream);
                ce = cudaStreamEndCapture(stream, &g);
                if (le != cudaSuccess) ce = le;
            }
            if (ce == cudaSuccess) ce = cudaGraphInstantiate(&ge, g, 0);
            if (g) cudaGraphDestroy(g);
            if (ce == cudaSuccess) {
                it = e->graphs.emplace(n_steps, ge).first;
            } else {
                cudaGetLastError();  // clear; fall back to direct launches
                e->graphs_ok = false;
            }
        }
        if (e->graphs_ok) {
            ce = cudaGraphLaunch(it->second, stream);
            if (ce != cudaSuccess) { set_last_error("cudaGraphLaunch", ce); return PHS_ERR_CUDA; }
            launched = true;
        }
    }
    if (!launched) {
        ce = launch_waves<T>(e, n_steps, stream);
        if (ce != cudaSuccess) { set_last_error("launch step_kernel", ce); return PHS_ERR_CUDA; }
    }
    e->launches += (long long)e->waves.size();
    if (!sync) return PHS_OK;
    PHS_CUDA_TRY(cudaStreamSynchronize(stream));
    unsigned int ab = 0;
    PHS_CUDA_TRY(cudaMemcpy(&ab, e->abort_word, sizeof(ab), cudaMemcpyDeviceToHost));
    if (ab) { e->broken = true; return PHS_ERR_TIMEOUT; }
    int worst = PHS_OK;
    for (int i : act) {
        InstHost& h = e->inst[i];
        PHS_CUDA_TRY(cudaMemcpy(&h.st_host, h.st, sizeof(InstState), cudaMemcpyDeviceToHost));
        if (h.st_host.step >= h.d.n_steps || h.st_host.status == PHS_ERR_NONFINITE) {
            if (!h.finished) e->dirty = true;
            h.finished = true;
        }
        if (h.st_host.status == PHS_ERR_NONFINITE) worst = PHS_ERR_NONFINITE;
        else if (h.st_host.status == PHS_WARN_NO_CONVERGE && worst == PHS_OK) worst = PHS_WARN_NO_CONVERGE;
    }
    return worst;
}

// Moves the arrays whose addresses the caller asked for out of the pool into
// cudaMalloc memory, which peers can be given access to and other processes a
// handle of; pool memory has neither.  Only then: three cudaMalloc and cudaFree
// calls per instance cost more than adding it otherwise does.  Where there is no
// memory for them the arrays stay in the pool.
void export_arrays(phs_engine* e, InstHost& h) {
    if (h.exported) return;
    DeviceGuard guard(e->device);
    // a stream capture that another thread has under way is not disturbed
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    const size_t es = (e->prec == PHS_PREC_F64) ? 8 : 4;
    void* old[3] = {h.u, h.hist_u, h.lat};
    const size_t bytes[3] = {(size_t)h.ldv * es, (size_t)std::max(h.d.n_samples, 1) * h.n * es, (size_t)h.ldv * 4};
    void* p[3] = {nullptr, nullptr, nullptr};
    cudaError_t ce = cudaDeviceSynchronize();
    for (int i = 0; i < 3 && ce == cudaSuccess; ++i) ce = cudaMalloc(&p[i], bytes[i]);
    for (int i = 0; i < 3 && ce == cudaSuccess; ++i) ce = cudaMemcpyAsync(p[i], old[i], bytes[i], cudaMemcpyDeviceToDevice, 0);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(0);
    if (ce == cudaSuccess) {
        for (void* q : old) dev_free(q, 0);
        h.u = p[0];
        h.hist_u = p[1];
        h.lat = (int32_t*)p[2];
        h.exported = true;
        e->dirty = true;       // the launch plan holds the old addresses
    } else {
        for (void* q : p) cudaFree(q);
        cudaGetLastError();
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
}

}  // namespace

// ====================================================================== C ABI
extern "C" {

int phs_device_query(int precision, int* sm_count, int* ctas_per_sm) {
    int dev = 0;
    PHS_CUDA_TRY(cudaGetDevice(&dev));
    int sms = 0;
    PHS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int occ = 0;
    int rc = (precision == PHS_PREC_F64) ? occupancy_for<double>(&occ, kDefaultF64)
                                         : occupancy_for<float>(&occ, kDefaultF32);
    if (rc != PHS_OK) return rc;
    if (sm_count) *sm_count = sms;
    if (ctas_per_sm) *ctas_per_sm = occ;
    return PHS_OK;
}

int phs_engine_create(int precision, phs_engine** out) {
    if (!out || (precision != PHS_PREC_F32 && precision != PHS_PREC_F64)) return PHS_ERR_BAD_ARG;
    phs_engine* e = new phs_engine();
    e->prec = precision;
    cudaError_t ce = cudaGetDevice(&e->device);
    if (ce == cudaSuccess) ce = cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, e->device);
    if (ce == cudaSuccess) ce = dev_alloc((void**)&e->abort_word, sizeof(unsigned int), 0);
    if (ce == cudaSuccess) ce = cudaMemset(e->abort_word, 0, sizeof(unsigned int));
    if (ce != cudaSuccess) {
        set_last_error("phs_engine_create", ce);
        dev_free(e->abort_word, 0);
        delete e;
        return PHS_ERR_CUDA;
    }
    pool_update(1);
    *out = e;
    return PHS_OK;
}

int phs_engine_destroy(phs_engine* e) {
    if (!e) return PHS_ERR_BAD_ARG;
    DeviceGuard guard(e->device);
    cudaDeviceSynchronize();
    drop_graphs(e);
    for (auto& h : e->inst)
        if (h.used) free_inst(h);
    dev_free(e->abort_word, 0);
    dev_free(e->d_desc, 0);
    dev_free(e->d_map, 0);
    pool_update(-1);
    cudaStreamSynchronize(0);   // the driver has what the pool does not keep
    delete e;
    return PHS_OK;
}

int phs_instance_add(phs_engine* e, const phs_instance_desc* d, int* slot) {
    if (!e || !d || !slot) return PHS_ERR_BAD_ARG;
    return e->prec == PHS_PREC_F64 ? add_instance<double>(e, d, slot) : add_instance<float>(e, d, slot);
}

int phs_instance_remove(phs_engine* e, int slot) {
    if (!e || slot < 0 || slot >= (int)e->inst.size() || !e->inst[slot].used) return PHS_ERR_BAD_ARG;
    DeviceGuard guard(e->device);
    cudaDeviceSynchronize();
    free_inst(e->inst[slot]);
    pool_update(0);
    cudaStreamSynchronize(0);   // the driver has what the pool does not keep
    e->dirty = true;
    e->auto_left = 2;
    e->auto_mark = e->launches;
    return PHS_OK;
}

int phs_instance_info_get(phs_engine* e, int slot, phs_instance_info* info) {
    if (!e || !info || slot < 0 || slot >= (int)e->inst.size() || !e->inst[slot].used) return PHS_ERR_BAD_ARG;
    InstHost& h = e->inst[slot];
    PHS_CUDA_TRY(cudaMemcpy(&h.st_host, h.st, sizeof(InstState), cudaMemcpyDeviceToHost));
    info->n_voxel = h.n;
    info->step = h.st_host.step;
    info->n_steps = h.d.n_steps;
    info->samples = h.st_host.id_save;
    info->status = h.st_host.status;
    info->arnoldi_steps = h.st_host.arnoldi;
    info->solves = h.st_host.solves;
    info->max_arnoldi = h.st_host.max_arnoldi;
    info->nonconverged = h.st_host.nonconv;
    info->arnoldi_sq = h.st_host.arnoldi_sq;
    return PHS_OK;
}

int phs_engine_advance(phs_engine* e, int64_t n_steps, int ctas_per_sm, void* stream, int sync) {
    if (!e || n_steps < 0) return PHS_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    return e->prec == PHS_PREC_F64 ? advance_impl<double>(e, n_steps, ctas_per_sm, s, sync != 0)
                                   : advance_impl<float>(e, n_steps, ctas_per_sm, s, sync != 0);
}

int phs_instance_read_history(phs_engine* e, int slot, int32_t s0, int32_t count, void* u_dst, void* h_dst) {
    if (!e || slot < 0 || slot >= (int)e->inst.size() || !e->inst[slot].used) return PHS_ERR_BAD_ARG;
    InstHost& h = e->inst[slot];
    if (s0 < 0 || count < 0 || s0 + count > h.d.n_samples) return PHS_ERR_BAD_ARG;
    const size_t es = (e->prec == PHS_PREC_F64) ? 8 : 4;
    const size_t off = (size_t)s0 * h.n * es, bytes = (size_t)count * h.n * es;
    PHS_CUDA_TRY(cudaDeviceSynchronize());
    if (u_dst && bytes) PHS_CUDA_TRY(cudaMemcpy(u_dst, (char*)h.hist_u + off, bytes, cudaMemcpyDeviceToHost));
    if (h_dst && bytes) {
        if (!h.hist_h) return PHS_ERR_STATE;
        PHS_CUDA_TRY(cudaMemcpy(h_dst, (char*)h.hist_h + off, bytes, cudaMemcpyDeviceToHost));
    }
    return PHS_OK;
}

int phs_instance_read_state(phs_engine* e, int slot, void* u_dst, void* h_dst, int32_t* lat_dst) {
    if (!e || slot < 0 || slot >= (int)e->inst.size() || !e->inst[slot].used) return PHS_ERR_BAD_ARG;
    InstHost& h = e->inst[slot];
    PHS_CUDA_TRY(cudaDeviceSynchronize());
    PHS_CUDA_TRY(cudaMemcpy(&h.st_host, h.st, sizeof(InstState), cudaMemcpyDeviceToHost));
    const size_t es = (e->prec == PHS_PREC_F64) ? 8 : 4;
    if (u_dst) PHS_CUDA_TRY(cudaMemcpy(u_dst, h.u, (size_t)h.n * es, cudaMemcpyDeviceToHost));
    if (h_dst) {
        const void* hc = h.st_host.hbuf ? h.h1 : h.h0;
        PHS_CUDA_TRY(cudaMemcpy(h_dst, hc, (size_t)h.n * es, cudaMemcpyDeviceToHost));
    }
    if (lat_dst) PHS_CUDA_TRY(cudaMemcpy(lat_dst, h.lat, (size_t)h.n * 4, cudaMemcpyDeviceToHost));
    return PHS_OK;
}

int phs_instance_device_views(phs_engine* e, int slot, void** u, void** hist_u, int32_t** lat) {
    if (!e || slot < 0 || slot >= (int)e->inst.size() || !e->inst[slot].used) return PHS_ERR_BAD_ARG;
    const InstHost& h = e->inst[slot];
    if (u) *u = h.u;
    if (hist_u) *hist_u = h.hist_u;
    if (lat) *lat = h.lat;
    return PHS_OK;
}

int phs_instance_device_ptrs(phs_engine* e, int slot, void** u, void** hist_u, int32_t** lat) {
    if (!e || slot < 0 || slot >= (int)e->inst.size() || !e->inst[slot].used) return PHS_ERR_BAD_ARG;
    InstHost& h = e->inst[slot];
    export_arrays(e, h);
    if (u) *u = h.u;
    if (hist_u) *hist_u = h.hist_u;
    if (lat) *lat = h.lat;
    return PHS_OK;
}

int64_t phs_engine_launch_count(phs_engine* e) { return e ? e->launches : -1; }

int phs_engine_rebalance(phs_engine* e) {
    if (!e) return PHS_ERR_BAD_ARG;
    PHS_CUDA_TRY(cudaDeviceSynchronize());
    for (auto& h : e->inst) {
        if (!h.used) continue;
        PHS_CUDA_TRY(cudaMemcpy(&h.st_host, h.st, sizeof(InstState), cudaMemcpyDeviceToHost));
        const long long ds = h.st_host.step - h.ref_step;
        if (ds > 0) h.kavg = (double)(h.st_host.arnoldi - h.ref_arnoldi) / (double)ds;
        h.ref_step = h.st_host.step;
        h.ref_arnoldi = h.st_host.arnoldi;
        // measured cost: the team's time per step times its CTAs
        h.weight = 0.0;
        if (h.prof) {
            unsigned long long pf[kProfSlots];
            PHS_CUDA_TRY(cudaMemcpy(pf, h.prof, sizeof(pf), cudaMemcpyDeviceToHost));
            const unsigned long long steps = pf[PF_STEPS] - h.prof_ref[PF_STEPS];
            unsigned long long ns = 0;
            for (int i = 0; i <= PF_RHS1; ++i) ns += pf[i] - h.prof_ref[i];
            if (steps > 0 && h.team > 0) h.weight = (double)ns / (double)steps * (double)h.team;
            for (int i = 0; i < kProfSlots; ++i) h.prof_ref[i] = pf[i];
        }
    }
    e->dirty = true;
    return PHS_OK;
}

int phs_instance_profile(phs_engine* e, int slot, uint64_t* out16) {
    if (!e || !out16 || slot < 0 || slot >= (int)e->inst.size() || !e->inst[slot].used) return PHS_ERR_BAD_ARG;
    InstHost& h = e->inst[slot];
    if (!h.prof) return PHS_ERR_STATE;
    PHS_CUDA_TRY(cudaDeviceSynchronize());
    PHS_CUDA_TRY(cudaMemcpy(out16, h.prof, kProfSlots * sizeof(uint64_t), cudaMemcpyDeviceToHost));
    return PHS_OK;
}

int phs_instance_table_bytes(phs_engine* e, int slot, int32_t* bytes_per_voxel) {
    if (!e || !bytes_per_voxel || slot < 0 || slot >= (int)e->inst.size() || !e->inst[slot].used)
        return PHS_ERR_BAD_ARG;
    *bytes_per_voxel = (e->compact_nb && e->inst[slot].nbr) ? 8 : 24;
    return PHS_OK;
}

int phs_step_variants(int precision, int32_t* count, int32_t* min_ctas_per_sm, int32_t* max_regs) {
    if (precision != PHS_PREC_F32 && precision != PHS_PREC_F64) return PHS_ERR_BAD_ARG;
    const int nv = precision == PHS_PREC_F64 ? kNumF64 : kNumF32;
    if (count) *count = nv;
    for (int v = 0; v < nv; ++v) {
        if (min_ctas_per_sm) min_ctas_per_sm[v] = precision == PHS_PREC_F64 ? kMinbF64[v] : kMinbF32[v];
        if (max_regs) {
            cudaFuncAttributes a{};
            const void* fn = precision == PHS_PREC_F64 ? step_fn<double>(v) : step_fn<float>(v);
            max_regs[v] = (cudaFuncGetAttributes(&a, fn) == cudaSuccess) ? a.numRegs : -1;
        }
    }
    return PHS_OK;
}

namespace {
// Phase timers on or off for every instance (counters reset).
int set_profile(phs_engine* e, bool on) {
    cudaDeviceSynchronize();
    e->profile = on;
    for (auto& h : e->inst) {
        if (!h.used) continue;
        if (e->profile && !h.prof) {
            if (dev_alloc((void**)&h.prof, kProfSlots * sizeof(unsigned long long), 0) != cudaSuccess)
                return PHS_ERR_OOM;
        }
        if (h.prof) cudaMemset(h.prof, 0, kProfSlots * sizeof(unsigned long long));
        if (!e->profile && h.prof) { dev_free(h.prof, 0); h.prof = nullptr; }
        for (int i = 0; i < kProfSlots; ++i) h.prof_ref[i] = 0;
    }
    e->dirty = true;
    return PHS_OK;
}
}  // namespace

int phs_step_variant_vpt(int precision, int32_t count, int32_t* vpt) {
    if (precision != PHS_PREC_F32 && precision != PHS_PREC_F64) return PHS_ERR_BAD_ARG;
    const int nv = precision == PHS_PREC_F64 ? kNumF64 : kNumF32;
    if (count < nv || !vpt) return PHS_ERR_BAD_ARG;
    for (int v = 0; v < nv; ++v) vpt[v] = precision == PHS_PREC_F64 ? kVptF64 : kVptOfF32[v];
    return PHS_OK;
}

int phs_step_variant_layout(int precision, int32_t count, int32_t* ring_bytes, int32_t* compact_table) {
    if (precision != PHS_PREC_F32 && precision != PHS_PREC_F64) return PHS_ERR_BAD_ARG;
    const int nv = precision == PHS_PREC_F64 ? kNumF64 : kNumF32;
    if (count < nv) return PHS_ERR_BAD_ARG;
    for (int v = 0; v < nv; ++v) {
        const bool f32 = precision == PHS_PREC_F32;
        if (ring_bytes) ring_bytes[v] = f32 ? kRingF32[v] : 0;
        // staged variants read the compact table of every instance that has one
        if (compact_table) compact_table[v] = (f32 && (kTwinF32[v] >= 0 || kRingF32[v] > 0)) ? 1 : 0;
    }
    return PHS_OK;
}

int phs_engine_config(phs_engine* e, int key, int64_t value) {
    if (!e) return PHS_ERR_BAD_ARG;
    switch (key) {
        case PHS_CFG_VARIANT: {
            const int nv = e->prec == PHS_PREC_F64 ? kNumF64 : kNumF32;
            if (value < -1 || value >= nv) return PHS_ERR_BAD_ARG;
            if (e->variant != (int)value) {
                e->variant = (int)value;
                e->dirty = true;
            }
            return PHS_OK;
        }
        case PHS_CFG_CTAS_PER_SM:
            if (value < 0 || value > 32) return PHS_ERR_BAD_ARG;
            e->default_cps = (int)value;
            return PHS_OK;
        case PHS_CFG_AUTO_BALANCE:
            e->auto_balance = value != 0;
            return PHS_OK;
        case PHS_CFG_TEST_TEAM_OVERCOUNT:
            e->test_overcount = value != 0;
            e->dirty = true;
            return PHS_OK;
        case PHS_CFG_PROFILE:
            // the caller's setting wins over the automatic balancing's
            e->auto_prof = false;
            return set_profile(e, value != 0);
        case PHS_CFG_GROUP_SUMS:
            return PHS_OK;   // partial sums are always kept per group of tiles
        case PHS_CFG_COMPACT_NB:
            if (e->compact_nb != (value != 0)) {
                e->compact_nb = value != 0;
                e->dirty = true;
            }
            return PHS_OK;
        case PHS_CFG_WAVE_INSTANCES:
            if (value < 0 || value > (1 << 20)) return PHS_ERR_BAD_ARG;
            if (e->wave_instances != (int)value) {
                e->wave_instances = (int)value;
                e->dirty = true;
            }
            return PHS_OK;
        default:
            return PHS_ERR_BAD_ARG;
    }
}

int phs_simulate(const phs_instance_desc* desc, int precision, void* u_hist, void* h_hist, int32_t* lat,
                 int32_t* n_saved, phs_instance_info* info) {
    if (!desc) return PHS_ERR_BAD_ARG;
    phs_engine* e = nullptr;
    int rc = phs_engine_create(precision, &e);
    if (rc != PHS_OK) return rc;
    int slot = -1;
    rc = phs_instance_add(e, desc, &slot);
    if (rc != PHS_OK) { phs_engine_destroy(e); return rc; }
    // bounded launches keep each kernel short
    const long long chunk = 2000;
    int worst = PHS_OK;
    for (long long done = 0; done < desc->n_steps; done += chunk) {
        rc = phs_engine_advance(e, chunk, 0, nullptr, 1);
        if (rc == PHS_WARN_NO_CONVERGE) worst = rc;
        else if (rc != PHS_OK) { phs_engine_destroy(e); return rc; }
    }
    phs_instance_info inf{};
    rc = phs_instance_info_get(e, slot, &inf);
    if (rc == PHS_OK && n_saved) *n_saved = inf.samples;
    if (rc == PHS_OK && inf.samples > 0 && (u_hist || h_hist))
        rc = phs_instance_read_history(e, slot, 0, inf.samples, u_hist, desc->save_h ? h_hist : nullptr);
    if (rc == PHS_OK && lat) rc = phs_instance_read_state(e, slot, nullptr, nullptr, lat);
    if (info) *info = inf;
    phs_engine_destroy(e);
    if (rc != PHS_OK) return rc;
    if (inf.status == PHS_ERR_NONFINITE) return PHS_ERR_NONFINITE;
    return worst != PHS_OK ? worst : inf.status;
}

}  // extern "C"
