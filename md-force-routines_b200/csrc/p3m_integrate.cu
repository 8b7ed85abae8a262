// Integrator, thermostat, energies, n(q,t) and the optimal influence function.
//
// One velocity-Verlet step (velocity_verlet_p3m_ord6.py:5-26) is split around
// the force evaluation:
//   k_kick_drift   v += 0.5 a dt; x += v dt; single periodic wrap (:7-19),
//                  fused with the PP-cell / mesh-brick keys of the new x
//   ... sort, PP, PM ...
//   k_kick_finish  a = af (a_pp + Z E) (yukawa_p3m_ord6.py:21); v += 0.5 a dt
//                  (:24); per-block sums of v^2 in FP64
//   k_finish_drift both in one pass, where a captured sequence allows it
//   k_step_reduce  per replica K = kf sum v^2, T = K/kf/N, U = uf (U_pp + U_pm
//                  + U_self) (yukawa_p3m_ord6.py:23-24) and, in thermostat
//                  mode, the factor of thermostat_p3m_ord6.py:9-23
//   k_scale_vel    v *= factor (thermostat mode only)
// The position and velocity updates use explicitly rounded FP64 operations in
// the reference's order (no FMA contraction), so a step reproduces the
// reference's rounding.
#include "p3m_kernels.h"

namespace p3m {

__device__ __forceinline__ double kick(double v, double a, double dt)
{
    // v + 0.5*a*dt, evaluated as v + ((0.5*a)*dt)
    return __dadd_rn(v, __dmul_rn(__dmul_rn(0.5, a), dt));
}

__device__ __forceinline__ double wrap_once(double x, double L)
{
    // velocity_verlet_p3m_ord6.py:16-19: if x > Lmax: x -= L; if x < Lmin: x += L
    if (x > L) x = __dsub_rn(x, L);
    if (x < 0.0) x = __dadd_rn(x, L);
    return x;
}

// A particle's drift from its kicked velocity v: new position, rebuild and prune
// flags, brick key and arrival rank. Also the coordinates of the pair stage, at
// the slots of the last cell sort (a replica that rebuilds this step has them
// rewritten at its new slots by k_fix_cells): a pass of its own read the
// positions again at random (1e6 particles: 40 us).
struct DriftArgs {
    double *pos = nullptr;
    const double *pos_ref = nullptr, *pos_pref = nullptr;  // pos_pref: inner lists only
    int *brick_key = nullptr, *brick_rank = nullptr, *brick_count = nullptr;
    int has_mesh = 0;
    int *rebuild = nullptr, *prune = nullptr, *status = nullptr;
    const int *cell_slot = nullptr;
    void *xq = nullptr;
};

// What the drift reads, loaded before the pass's first store (the compiler keeps
// loads behind stores that could alias them).
struct DriftIn {
    double x[3], ref[3], pref[3];
    int slot;
    __device__ __forceinline__ DriftIn(const DriftArgs &A, int i) : slot(A.cell_slot[i])
    {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            x[d] = A.pos[3 * i + d];
            ref[d] = A.pos_ref[3 * i + d];
            pref[d] = A.pos_pref ? A.pos_pref[3 * i + d] : 0.0;
        }
    }
};

template <typename T>
__device__ __forceinline__ void drift(const DriftArgs &A, const RepDev &R, int r, int i, const DriftIn &in,
                                      const double *v)
{
    double x[3];
    double d2 = 0.0, d2p = 0.0;
    bool vfin = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        vfin = vfin && isfinite(v[d]);
        x[d] = wrap_once(__dadd_rn(in.x[d], __dmul_rn(v[d], R.dt)), R.L);
        A.pos[3 * i + d] = x[d];
        // displacement since the last list rebuild, minimum image
        double dd = x[d] - in.ref[d];
        dd = fma(-R.L, rint(dd * R.inv_L), dd);
        d2 = fma(dd, dd, d2);
        if (A.pos_pref) {  // and since the last inner-list build
            double dp = x[d] - in.pref[d];
            dp = fma(-R.L, rint(dp * R.inv_L), dp);
            d2p = fma(dp, dp, d2p);
        }
    }
    // a non-finite velocity (or acceleration) is reported as such; the
    // position it makes is also flagged by particle_keys below
    if (!vfin) raise_status(A.status, ST_NONFINITE);
    if (d2 > 0.25 * R.skin * R.skin && !A.rebuild[r]) atomicOr(A.rebuild + r, 1);
    if (A.pos_pref && d2p > 0.25 * R.pbuf * R.pbuf && !A.prune[r]) atomicOr(A.prune + r, 1);
    int b, rank = 0;
    particle_keys(R, x[0], x[1], x[2], A.has_mesh, nullptr, &b, A.status);
    if (b >= 0) rank = atomicAdd(&A.brick_count[b * BRICK_CNT_STRIDE], 1);
    // while the atomic returns
    ((typename Coord<T>::Q *)A.xq)[in.slot] = quantize<T>(x[0], x[1], x[2], R.inv_L, r);
    if (b >= 0) {
        A.brick_key[i] = b;
        A.brick_rank[i] = rank;
    }
}

template <typename T>
__global__ void k_kick_drift(const RepDev *__restrict__ reps, const int *__restrict__ prep,
                             double *__restrict__ vel, const double *__restrict__ acc, int ntot,
                             DriftArgs A)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ntot; i += gridDim.x * blockDim.x) {
        const int r = prep[i];
        const RepDev &R = reps[r];
        const DriftIn in(A, i);
        double v[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            v[d] = kick(vel[3 * i + d], acc[3 * i + d], R.dt);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) vel[3 * i + d] = v[d];
        drift<T>(A, R, r, i, in, v);
    }
}

// Replica-aligned particle blocks: block b belongs to replica r and covers
// particles p_off + (b - blk_off) * PBLK + [0, PBLK).
__device__ __forceinline__ int block_replica(const RepDev *reps, int nrep, int b)
{
    return find_rep(b, nrep, [&](int k) { return reps[k].blk_off; });
}

constexpr int SR_THREADS = 512;

// Sum of a replica's kinetic partials [b0, b1), in every thread of the block:
// entry k by thread k mod SR_THREADS, then a fixed tree, whatever the block size.
// red: SR_THREADS / 32 doubles.
template <int NT>
__device__ __forceinline__ double kin_sum(const double *__restrict__ kin_part, int b0, int b1, double *red)
{
    static_assert(SR_THREADS % NT == 0, "whole shares");
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
#pragma unroll
    for (int h = 0; h < SR_THREADS / NT; ++h) {
        double s = 0.0;
        for (int k = b0 + tid + h * NT; k < b1; k += SR_THREADS) s += kin_part[k];
        s = warp_sum(s);
        if (lane == 0) red[w + h * (NT / 32)] = s;
    }
    __syncthreads();
    return warp_sum(lane < SR_THREADS / 32 ? red[lane] : 0.0);
}

// The thermostat's factor after step `it`, from the sum of v^2
// (thermostat_p3m_ord6.py:15-23)
__device__ __forceinline__ double thermostat_factor(const RepDev &R, double s, int it)
{
    const double T = R.kf * s / R.kf / (double)R.n;
    return (it <= 1999) ? sqrt(R.t_desired / T) : sqrt((20.0 * R.t_desired / T - 1.0) / 20.0);
}

// k_kick_drift after a thermostat step of the same captured sequence: every
// block takes its replica's factor from the kinetic partials itself, so that the
// energy reduction, which does the same sum, runs beside this pass and not
// before it (2e3 particles 41.2 -> 39.3 us a step, twelve uneven replicas 631.2 ->
// 630.2). it: the finished step's index.
template <typename T>
__global__ void __launch_bounds__(PBLK)
k_rescale_drift(const RepDev *__restrict__ reps, int nrep, int nblk, double *__restrict__ vel,
                const double *__restrict__ acc, const double *__restrict__ kin_part,
                const int *__restrict__ it, DriftArgs A)
{
    __shared__ double red[SR_THREADS / 32];
    const int b = blockIdx.x, r = block_replica(reps, nrep, b);
    const RepDev &R = reps[r];
    const int i = R.p_off + (b - R.blk_off) * PBLK + threadIdx.x;
    const double s = kin_sum<PBLK>(kin_part, R.blk_off, r + 1 < nrep ? reps[r + 1].blk_off : nblk, red);
    if (i >= R.p_off + R.n) return;
    const DriftIn in(A, i);
    const double fact = thermostat_factor(R, s, *it);
    double v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d] = kick(__dmul_rn(vel[3 * i + d], fact), acc[3 * i + d], R.dt);
#pragma unroll
    for (int d = 0; d < 3; ++d) vel[3 * i + d] = v[d];
    drift<T>(A, R, r, i, in, v);
}

struct FinishArgs {
    const int *cell_slot = nullptr, *brick_slot = nullptr;
    const void *acc_pp = nullptr, *acc_pm = nullptr;
    int has_mesh = 0;
    double *vel = nullptr, *kin_part = nullptr;
    int *status = nullptr;
    int *rebuild = nullptr, *prune = nullptr;  // the finished step's flags; prune: inner lists only
    double *prune_count = nullptr, *rep_out = nullptr;
    int *counters = nullptr;  // set: [7] receives the step's index, for k_rescale_drift
};

// a = af (a_pp + Z E) of a particle
template <typename T>
__device__ __forceinline__ void combine(const FinishArgs &A, const RepDev &R, int i, double *a,
                                        double *ep_out)
{
    using T4 = typename V4<T>::t;
    const T4 ap = ((const T4 *)A.acc_pp)[A.cell_slot[i]];
    a[0] = (double)ap.x;
    a[1] = (double)ap.y;
    a[2] = (double)ap.z;
    if (A.has_mesh) {
        const T4 e = ((const T4 *)A.acc_pm)[A.brick_slot[i]];
        const double q = (double)e.w;
        const double E[3] = {(double)e.x, (double)e.y, (double)e.z};
#pragma unroll
        for (int d = 0; d < 3; ++d) a[d] = fma(q, E[d], a[d]);
        if (ep_out) {
            ep_out[3 * i + 0] = E[0];
            ep_out[3 * i + 1] = E[1];
            ep_out[3 * i + 2] = E[2];
        }
    }
    bool finite = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        a[d] = R.af * a[d];
        finite = finite && isfinite(a[d]);
    }
    if (!finite) raise_status(A.status, ST_NONFINITE);
}

// The lists of a step are built and used: count the builds (steps only) and
// clear the flags. One block.
__device__ __forceinline__ void settle_flags(const FinishArgs &A, int nrep, int do_kick)
{
    for (int k = threadIdx.x; k < nrep; k += PBLK) {
        const bool fr = A.rebuild[k] != 0;
        if (fr && do_kick) A.rep_out[8 * k + RO_REBUILDS] += 1.0;
        if (A.prune) {  // inner lists: count the builds that came without an outer rebuild
            if (A.prune[k] && !fr && do_kick) A.prune_count[k] += 1.0;
            A.prune[k] = 0;
        }
        A.rebuild[k] = 0;
    }
}

// acc = af (a_pp + Z E) for every particle; with do_kick the second half kick
// and the per-block FP64 sum of v^2. Block 0 settles the flags, which the next
// drift may raise again.
template <typename T>
__global__ void __launch_bounds__(PBLK)
k_kick_finish(const RepDev *__restrict__ reps, int nrep, FinishArgs A, double *__restrict__ acc,
              int do_kick, double *__restrict__ ep_out)
{
    __shared__ double red[32];
    const int b = blockIdx.x;
    if (b == 0) {
        settle_flags(A, nrep, do_kick);
        if (A.counters && threadIdx.x == 0) A.counters[7] = A.counters[2] + A.counters[0];
    }
    const int r = block_replica(reps, nrep, b);
    const RepDev &R = reps[r];
    const int i = R.p_off + (b - R.blk_off) * PBLK + threadIdx.x;
    double kin = 0.0;
    if (i < R.p_off + R.n) {
        double a[3], v[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] = do_kick ? A.vel[3 * i + d] : 0.0;
        combine<T>(A, R, i, a, ep_out);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            acc[3 * i + d] = a[d];
            if (do_kick) {
                v[d] = kick(v[d], a[d], R.dt);
                A.vel[3 * i + d] = v[d];
                kin = fma(v[d], v[d], kin);
            }
        }
    }
    const double t = block_sum(kin, red);
    if (threadIdx.x == 0) A.kin_part[b] = t;
}

// A step's end and the next one's beginning in one pass, for steps of one
// captured sequence with nothing between them that needs all particles (NVE, no
// snapshots): second half kick, sum of v^2, first half kick, drift. The
// acceleration stays in registers. The two steps' flags are different arrays (F's
// are settled, D's raised). Bound: latency in small systems -- a kernel and its
// edge less on the serial chain -- and memory in large ones (us a step, two passes
// / one: 1e4 particles 50.0 / 47.4, FP64 74.0 / 71.3, 20 x 1e4 403 / 400, 1e5
// 271.1 / 269.6, 1e6 1775 / 1746).
template <typename T>
__global__ void __launch_bounds__(PBLK)
k_finish_drift(const RepDev *__restrict__ reps, int nrep, FinishArgs F, DriftArgs D)
{
    __shared__ double red[32];
    const int b = blockIdx.x;
    if (b == 0) settle_flags(F, nrep, 1);
    const int r = block_replica(reps, nrep, b);
    const RepDev &R = reps[r];
    const int i = R.p_off + (b - R.blk_off) * PBLK + threadIdx.x;
    double kin = 0.0;
    if (i < R.p_off + R.n) {
        const DriftIn in(D, i);
        double a[3], v[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] = F.vel[3 * i + d];
        combine<T>(F, R, i, a, nullptr);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            v[d] = kick(v[d], a[d], R.dt);
            kin = fma(v[d], v[d], kin);
            v[d] = kick(v[d], a[d], R.dt);
            F.vel[3 * i + d] = v[d];
        }
        drift<T>(D, R, r, i, in, v);
    }
    const double t = block_sum(kin, red);
    if (threadIdx.x == 0) F.kin_part[b] = t;
}

// Energies, temperature and the thermostat factor, one block per replica; one
// row of the energy ring; the last block to finish advances the step counters.
// mode: 0 NVE, 1 thermostat, 2 force only (no kinetic terms). Latency-bound, on
// the step's serial tail: the partials are summed by the block's threads (entry
// k by thread k mod SR_THREADS, then a fixed tree -- the same order whatever the
// batch). One block for all replicas, a warp each, took 5.4 us for 1e4 particles
// against 4.0, 7.4 for 20 x 1e4 against 5.9, 30 for 1e6 against 8.9.
__global__ void __launch_bounds__(SR_THREADS)
k_step_reduce(const RepDev *__restrict__ reps, int nrep, int nblk,
              const double *__restrict__ kin_part, double *__restrict__ rep_out,
              int mode, int *__restrict__ counters, double *__restrict__ ring,
              int ring_cap, int recorded, int snap_interval, int snap_cap, int *status,
              StepSums sums)
{
    // counters: [0] steps since the run started, [1] energy-ring position,
    // [2] step index of the run's first step (thermostat_p3m_ord6.py:15 tests
    // it <= 1999), [3] n(q,t) rows recorded, [4] snapshots taken, [5] the
    // snapshot slot this step writes (-1: none), [6] blocks finished, [7] see
    // k_kick_finish
    __shared__ double part[3][SR_THREADS / 32];
    const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int it = counters[2] + counters[0];
    const int step = counters[1];
    const RepDev &R = reps[r];
    const bool last = r + 1 == nrep;
    double t = 0.0, tm = 0.0;
    if (sums.u_pp_part) {  // (k_reduce_pp and k_reduce_pm outside a step)
        const int b0 = R.pp_blk_off, b1 = last ? sums.pp_nblk : reps[r + 1].pp_blk_off;
        for (int k = b0 + tid; k < b1; k += SR_THREADS) t += sums.u_pp_part[k];
        if (R.M > 0) {
            const int c0 = R.wc_off, c1 = last ? sums.wc_total : reps[r + 1].wc_off;
            const int p0 = sums.wc_total + R.wp_off,
                      p1 = sums.wc_total + (last ? sums.wp_total : reps[r + 1].wp_off);
            for (int k = c0 + tid; k < c1; k += SR_THREADS) tm += sums.u_pm_part[k];
            for (int k = p0 + tid; k < p1; k += SR_THREADS) tm += sums.u_pm_part[k];
        }
    }
    t = warp_sum(t);
    tm = warp_sum(tm);
    if (lane == 0) {
        part[0][w] = t;
        part[1][w] = tm;
    }
    const double s = kin_sum<SR_THREADS>(kin_part, R.blk_off, last ? nblk : reps[r + 1].blk_off, part[2]);
    if (w != 0) return;
    constexpr int NW = SR_THREADS / 32;
    t = warp_sum(lane < NW ? part[0][lane] : 0.0);
    tm = warp_sum(lane < NW ? part[1][lane] : 0.0);
    if (lane != 0) return;
    double *o = rep_out + 8 * r;
    const double u_pp = sums.u_pp_part ? 0.5 * t : o[RO_UPP];
    const double u_pm = sums.u_pp_part ? 0.5 * tm : o[RO_UPM];
    const double u_self = -R.n * R.alpha / 1.7724538509055160273;
    const double U = R.uf * (u_pp + u_pm + u_self);
    const double K = R.kf * s;
    const double T = K / R.kf / (double)R.n;
    const double fact = mode == 1 ? thermostat_factor(R, s, it) : 1.0;
    if (!isfinite(U)) raise_status(status, ST_NONFINITE);
    o[RO_UPP] = u_pp;
    o[RO_UPM] = u_pm;
    o[RO_USELF] = u_self;
    o[RO_U] = U;
    o[RO_K] = K;
    o[RO_T] = T;
    o[RO_FACT] = fact;
    if (ring && ring_cap > 0) {
        double *row = ring + ((long long)(step % ring_cap) * nrep + r) * 4;
        row[0] = U;
        row[1] = K;
        row[2] = T;
        row[3] = fact;
    }
    if (mode == 2) return;
    // every block has read the counters once all have taken a ticket
    if (nrep > 1) {
        __threadfence();
        if (atomicAdd(&counters[6], 1) != nrep - 1) return;
        counters[6] = 0;
    }
    counters[0] = it - counters[2] + 1;
    counters[1] = step + 1;
    if (recorded) counters[3] += 1;
    // a snapshot after step `it` when (it + 1) % interval == 0, as the
    // reference writes its files (yukawa_MD_p3m_ord6.py:222)
    if (snap_interval > 0 && (it + 1) % snap_interval == 0) {
        counters[5] = counters[4] % snap_cap;
        counters[4] += 1;
    } else {
        counters[5] = -1;
    }
}

// The state after this step, [slot][particle][pos, vel, acc] (the rows of
// yukawa_MD_p3m_ord6.py:223), into the slot k_step_reduce chose; steps[slot]
// = the step index.
__global__ void k_snapshot(const double *__restrict__ pos, const double *__restrict__ vel,
                           const double *__restrict__ acc, int ntot,
                           const int *__restrict__ counters, double *__restrict__ snap,
                           int *__restrict__ steps)
{
    const int slot = counters[5];
    if (slot < 0) return;
    double *dst = snap + (long long)slot * ntot * 9;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ntot; i += gridDim.x * blockDim.x) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            dst[9 * (long long)i + c] = pos[3 * (long long)i + c];
            dst[9 * (long long)i + 3 + c] = vel[3 * (long long)i + c];
            dst[9 * (long long)i + 6 + c] = acc[3 * (long long)i + c];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) steps[slot] = counters[2] + counters[0] - 1;
}

__global__ void k_set_flags(int *flag, int n, int value)
{
    for (int r = threadIdx.x; r < n; r += blockDim.x) flag[r] = value;
}

__global__ void k_set_counters(int *counters, int run_step, int ring_pos, int it0)
{
    if (run_step >= 0) counters[0] = run_step;
    if (ring_pos >= 0) {
        counters[1] = ring_pos;
        counters[3] = ring_pos;
    }
    counters[2] = it0;
}

// out[i] = scale (use_pp a_pp + use_pm Z E) in original particle order; ep_out
// (optional) receives E at the particle.
template <typename T>
__global__ void k_combine(const RepDev *__restrict__ reps, const int *__restrict__ prep,
                          const int *__restrict__ cell_slot, const int *__restrict__ brick_slot,
                          const typename V4<T>::t *__restrict__ acc_pp,
                          const typename V4<T>::t *__restrict__ acc_pm, int use_pp, int use_pm,
                          int scale_af, double *__restrict__ out, double *__restrict__ ep_out,
                          int ntot, int *status)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ntot; i += gridDim.x * blockDim.x) {
        double a[3] = {0.0, 0.0, 0.0};
        if (use_pp) {
            const typename V4<T>::t ap = acc_pp[cell_slot[i]];
            a[0] = (double)ap.x;
            a[1] = (double)ap.y;
            a[2] = (double)ap.z;
        }
        if (use_pm) {
            const typename V4<T>::t e = acc_pm[brick_slot[i]];
            const double q = (double)e.w;
            a[0] = a[0] + q * (double)e.x;
            a[1] = a[1] + q * (double)e.y;
            a[2] = a[2] + q * (double)e.z;
            if (ep_out) {
                ep_out[3 * i + 0] = (double)e.x;
                ep_out[3 * i + 1] = (double)e.y;
                ep_out[3 * i + 2] = (double)e.z;
            }
        }
        const double f = scale_af ? reps[prep[i]].af : 1.0;
        out[3 * i + 0] = scale_af ? f * a[0] : a[0];
        out[3 * i + 1] = scale_af ? f * a[1] : a[1];
        out[3 * i + 2] = scale_af ? f * a[2] : a[2];
        if (!(isfinite(a[0]) && isfinite(a[1]) && isfinite(a[2]))) raise_status(status, ST_NONFINITE);
    }
}

__global__ void k_scale_vel(const RepDev *__restrict__ reps, const int *__restrict__ prep,
                            const double *__restrict__ rep_out, double *__restrict__ vel, int ntot)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ntot; i += gridDim.x * blockDim.x) {
        const double f = rep_out[8 * prep[i] + RO_FACT];
        vel[3 * i + 0] *= f;
        vel[3 * i + 1] *= f;
        vel[3 * i + 2] *= f;
    }
}

// n(q,t) partial sums: per replica-aligned block of NQ_PPT * PBLK particles,
// for each wave number q_m = m 2 pi / L (m = qmult[iq]) and axis,
// sum_i exp(-i q x_i) (yukawa_MD_p3m_ord6.py:215-219). Each thread sums
// NQ_PPT particles, a warp its 32 threads' sums (in the bulk precision T: a
// warp's total holds 32 NQ_PPT terms), and the block its warps' totals in
// FP64. The phase is reduced in FP64
// as frac(m x / L) before the sine/cosine of the bulk precision T; when the
// multiples are 1, 2, ..., nq (`consecutive`), exp(-i m theta) follows from
// exp(-i theta) by complex multiplication instead.
constexpr int NQ_PPT = 4;

template <typename T>
__device__ __forceinline__ void sincospi_t(double two_t, T *s, T *c)
{
    if (sizeof(T) == 4) {
        float sf, cf;
        sincospif((float)two_t, &sf, &cf);
        *s = (T)sf;
        *c = (T)cf;
    } else {
        double sd, cd;
        sincospi(two_t, &sd, &cd);
        *s = (T)sd;
        *c = (T)cd;
    }
}

// Sum over the 32 lanes of a warp of eight values v[0..7] per lane, by
// recursive halving: at each of the first three levels a lane keeps half of
// its values, sends the other half to its partner (lane ^ 16, ^ 8, ^ 4) and
// adds the partner's copy of the half it keeps; two butterfly levels finish
// the one value left. Lane l returns the total of value (l >> 2) & 7. Nine
// shuffles for eight sums (five per value in a plain butterfly), in a fixed
// order.
template <typename T>
__device__ __forceinline__ T warp_sum8(const T (&v)[8])
{
    const int lane = threadIdx.x & 31;
    T a[4], b[2];
    const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const T send = h4 ? v[i] : v[i + 4];
        a[i] = (h4 ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const T send = h3 ? a[i] : a[i + 2];
        b[i] = (h3 ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    const T send = h2 ? b[0] : b[1];
    T c = (h2 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, send, 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
    return c;
}

template <typename T, bool consecutive>
__global__ void __launch_bounds__(PBLK)
k_nqt_partial(const RepDev *__restrict__ reps, int nrep, const double *__restrict__ pos,
              const double *__restrict__ qmult, int nq, double *__restrict__ part)
{
    extern __shared__ double nsm[];  // [nwarps][nq*6]
    const int b = blockIdx.x;
    const int r = find_rep(b, nrep, [&](int k) { return reps[k].nq_blk_off; });
    const RepDev &R = reps[r];
    const int first = R.p_off + (b - R.nq_blk_off) * (PBLK * NQ_PPT);
    const int end = R.p_off + R.n;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double xl[NQ_PPT][3];
    bool have[NQ_PPT];
#pragma unroll
    for (int m = 0; m < NQ_PPT; ++m) {
        const int i = first + threadIdx.x + m * PBLK;
        have[m] = i < end;
#pragma unroll
        for (int d = 0; d < 3; ++d) xl[m][d] = have[m] ? pos[3 * i + d] * R.inv_L : 0.0;
    }
    // per-particle base rotation exp(-i 2 pi x/L) for the recurrence; a
    // missing particle rotates by 1 and is weighted by 0
    T c1[NQ_PPT][3], s1[NQ_PPT][3], cm[NQ_PPT][3], sm[NQ_PPT][3], wt[NQ_PPT];
#pragma unroll
    for (int m = 0; m < NQ_PPT; ++m) {
        wt[m] = have[m] ? (T)1 : (T)0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            T st = (T)0, ct = (T)1;
            if constexpr (consecutive) {
                const double t = xl[m][d] - floor(xl[m][d]);
                sincospi_t<T>(2.0 * t, &st, &ct);
            }
            c1[m][d] = ct;
            s1[m][d] = -st;
            cm[m][d] = (T)1;
            sm[m][d] = (T)0;
        }
    }
    for (int iq = 0; iq < nq; ++iq) {
        const double mq = consecutive ? 0.0 : qmult[iq];
        T acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = (T)0;
#pragma unroll
        for (int m = 0; m < NQ_PPT; ++m) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                T c, sn;
                if constexpr (consecutive) {
                    // exp(-i (k+1) theta) = exp(-i k theta) exp(-i theta)
                    const T nc = cm[m][d] * c1[m][d] - sm[m][d] * s1[m][d];
                    const T ns = cm[m][d] * s1[m][d] + sm[m][d] * c1[m][d];
                    cm[m][d] = nc;
                    sm[m][d] = ns;
                    c = nc;
                    sn = ns;
                } else {
                    double t = mq * xl[m][d];
                    t = t - floor(t);
                    T st, ct;
                    sincospi_t<T>(2.0 * t, &st, &ct);
                    c = ct;
                    sn = -st;
                }
                acc[2 * d + 0] += wt[m] * c;
                acc[2 * d + 1] += wt[m] * sn;
            }
        }
        // lane l holds the warp's total of value (l >> 2) & 7 (6, 7: padding)
        const T tot = warp_sum8<T>(acc);
        const int k = (lane >> 2) & 7;
        if ((lane & 3) == 0 && k < 6) nsm[w * nq * 6 + iq * 6 + k] = (double)tot;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nq * 6; k += blockDim.x) {
        double t = 0.0;
        for (int ww = 0; ww < nw; ++ww) t += nsm[ww * nq * 6 + k];
        part[(long long)b * nq * 6 + k] = t;
    }
}

// Per replica: sum the block partials into out[r][nq][3] complex (re, im).
// Block (r, c) sums values 32 c .. 32 c + 31 of replica r: warp w adds the
// partials of blocks b0 + w, b0 + w + 8, ... (lane = value), then the eight
// warp sums are added in warp order -- a fixed order, so the result does not
// depend on timing; a large replica's thousand partial blocks are summed by
// eight warps instead of one thread per value.
constexpr int NQR_WARPS = 8;

__global__ void __launch_bounds__(NQR_WARPS * 32)
k_nqt_reduce(const RepDev *__restrict__ reps, int nrep, int nblk,
             const double *__restrict__ part, int nq, double *__restrict__ out,
             const int *__restrict__ counters, int ring_cap)
{
    __shared__ double wsum[NQR_WARPS][32];
    const int r = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nv = nq * 6, k = blockIdx.y * 32 + lane;
    const RepDev &R = reps[r];
    const int b0 = R.nq_blk_off, b1 = (r + 1 < nrep) ? reps[r + 1].nq_blk_off : nblk;
    double s = 0.0;
    if (k < nv)
        for (int bb = b0 + w; bb < b1; bb += NQR_WARPS) s += part[(long long)bb * nv + k];
    wsum[w][lane] = s;
    __syncthreads();
    if (w == 0 && k < nv) {
        double t = 0.0;
        for (int j = 0; j < NQR_WARPS; ++j) t += wsum[j][lane];
        double *o = out;
        if (counters) {
            // ring layout [row][replica][nq][3][2]; this step's row
            const int step = counters[3] % ring_cap;
            o = out + (long long)step * nrep * nv;
        }
        o[(long long)r * nv + k] = t;
    }
}

// ---------------------------------------------------------------------------
// Optimal influence function (yukawa_gf_opt.py:5-98), FP64, fftshifted layout.
// ---------------------------------------------------------------------------
// On a cubic mesh G does not change when wave-vector components are permuted
// or change sign (the alias range -m .. m is symmetric; the Nyquist component
// of an even mesh has one sign only), so it is summed once per triple i <= j <=
// k of component sizes -- 6545 of the 262144 points of a 64^3 mesh -- and
// written to all its images. The Gaussian, U^2p and k k_m of a term are
// products or sums of one factor per axis, tabulated per triple; what is left
// per alias is a division. GF_LANES lanes share a triple: lane a takes the
// aliases az = a, a + GF_LANES, ... and a fixed shuffle tree adds them.
// One mesh of 64^3 with three aliases takes 28 us; with every point and an
// exponential per alias it took 717.
constexpr int GF_MAXA = 15;    // 2 * m_alias + 1 <= 15
constexpr int GF_LANES = 8;
constexpr int GF_THREADS = 256;
constexpr int GF_TRIPLES = GF_THREADS / GF_LANES;  // triples per block

// sizes of one component: 0 .. M/2 (even M), 0 .. (M-1)/2 (odd M)
static __host__ __device__ long long gf_triples(int M)
{
    const long long U = M / 2 + 1;
    return U * (U + 1) * (U + 2) / 6;
}

// exp(-(x / 2 alpha)^2): the rounding of the argument, which the exponential
// would multiply by the argument's size, is carried beside it. A Gaussian of
// zero also where x / alpha overflows.
__device__ __forceinline__ double gauss_factor(double x, double alpha)
{
    const double q = x / alpha, s = 0.25 * q * q;
    if (s >= 800.0) return 0.0;
    const double rest = fma(-q, alpha, x) / alpha;  // q + rest = x / alpha
    return exp(-s) * (1.0 - (fma(0.25 * q, q, -s) + 0.5 * q * rest));
}

// (sin x / x)^n. Around zero, the central aliases: from 1 - sin x / x, a short
// series, whose rounding is relative to that small difference -- the quotient's
// own would be raised to the n-th power.
__device__ __forceinline__ double sinc_power(double x, int n)
{
    if (fabs(x) <= 1.6) {
        const double t = x * x;
        double w = 1.0;
#pragma unroll
        for (int i = 12; i > 1; --i) w = fma(-t * (1.0 / (2 * i * (2 * i + 1))), w, 1.0);
        return exp(n * log1p(-t * (1.0 / 6.0) * w));
    }
    const double v = sin(x) / x;
    double up = 1.0;
    for (int q = 0; q < n; ++q) up *= v;
    return up;
}

__global__ void __launch_bounds__(GF_THREADS)
k_gf_opt(double kappa, double alpha, int p, int m, int M, double L, double *__restrict__ G_k,
         double *__restrict__ a_part)
{
    // per triple, axis and alias: k k_m, k_m^2, U^2p, exp(-k_m^2 / 4 alpha^2)
    __shared__ double tab[GF_TRIPLES][3][GF_MAXA][4];
    __shared__ double red[32];
    const double two_pi = 6.283185307179586477, four_pi = 12.566370614359172954;
    const double h = L / M;
    const int mid = M / 2;  // (M - 1) / 2 for odd M
    const int na = 2 * m + 1;
    const double kappa_sq = kappa * kappa;
    const int tl = threadIdx.x / GF_LANES, lane = threadIdx.x % GF_LANES;
    const long long t = blockIdx.x * (long long)GF_TRIPLES + tl;
    const bool have = t < gf_triples(M);
    // t = C(c + 2, 3) + C(b + 1, 2) + a with a <= b <= c
    int sz[3] = {0, 0, 0};
    if (have) {
        long long c = (long long)cbrt(6.0 * (double)t);
        while (c > 0 && c * (c + 1) * (c + 2) / 6 > t) --c;
        while ((c + 1) * (c + 2) * (c + 3) / 6 <= t) ++c;
        const long long r = t - c * (c + 1) * (c + 2) / 6;
        long long b = (long long)((sqrt(8.0 * (double)r + 1.0) - 1.0) * 0.5);
        while (b > 0 && b * (b + 1) / 2 > r) --b;
        while ((b + 1) * (b + 2) / 2 <= r) ++b;
        sz[0] = (int)(r - b * (b + 1) / 2);
        sz[1] = (int)b;
        sz[2] = (int)c;
    }
    const bool even = M % 2 == 0;
    double k_sq = 0.0;
    for (int d = 0; d < 3; ++d) {
        // the Nyquist component of an even mesh is negative
        const int s = even && sz[d] == M / 2 ? -sz[d] : sz[d];
        const double k = two_pi * s / L;
        k_sq += k * k;
        for (int a = lane; a < na; a += GF_LANES) {
            const double km = two_pi * (s + (double)(a - m) * M) / L;
            double *o = tab[tl][d][a];
            o[0] = k * km;
            o[1] = km * km;
            o[2] = sinc_power(0.5 * km * h, 2 * p);
            o[3] = gauss_factor(km, alpha);
        }
    }
    __syncwarp();
    double den = 0.0, num = 0.0;
    for (int az = lane; az < na; az += GF_LANES) {
        const double *tz = tab[tl][2][az];
        for (int ay = 0; ay < na; ++ay) {
            const double *ty = tab[tl][1][ay];
            const double dot = tz[0] + ty[0], q = kappa_sq + tz[1] + ty[1], u = tz[2] * ty[2],
                         g = tz[3] * ty[3];
            for (int ax = 0; ax < na; ++ax) {
                const double *tx = tab[tl][0][ax];
                const double u2 = u * tx[2];
                num += u2 * (g * tx[3] / (q + tx[1])) * (dot + tx[0]);
                den += u2;
            }
        }
    }
#pragma unroll
    for (int o = GF_LANES / 2; o > 0; o >>= 1) {
        num += __shfl_xor_sync(0xffffffffu, num, o);
        den += __shfl_xor_sync(0xffffffffu, den, o);
    }
    num *= four_pi * gauss_factor(kappa, alpha);
    double g = 0.0, acontrib = 0.0;
    if (have && k_sq != 0.0) {
        g = num / ((den * den) * k_sq);
        // number of mesh points the triple stands for
        int mult = sz[0] == sz[2] ? 1 : (sz[0] == sz[1] || sz[1] == sz[2] ? 3 : 6);
        for (int d = 0; d < 3; ++d) mult *= sz[d] > 0 && !(even && sz[d] == M / 2) ? 2 : 1;
        acontrib = mult * (num * num / ((den * den) * k_sq));
    }
    if (have) {
        // all six orders and eight sign choices (some coincide)
        for (int c = lane; c < 48; c += GF_LANES) {
            const int o = c % 6, sg = c / 6;
            const int i0 = o >> 1, i1 = (i0 + 1 + (o & 1)) % 3, i2 = 3 - i0 - i1;
            auto at = [&](int u, bool neg) { return neg || (even && u == M / 2) ? mid - u : mid + u; };
            const long long nx = at(sz[i0], sg & 1), ny = at(sz[i1], sg & 2), nz = at(sz[i2], sg & 4);
            G_k[(nz * M + ny) * M + nx] = g;
        }
    }
    const double ta = block_sum(lane == 0 ? acontrib : 0.0, red);
    if (threadIdx.x == 0) a_part[blockIdx.x] = ta;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static int pgrid(int n) { int g = (n + 255) / 256; return g < 1 ? 1 : (g > 148 * 16 ? 148 * 16 : g); }

static DriftArgs drift_args(const DevState &s)
{
    DriftArgs A;
    A.pos = s.pos;
    A.pos_ref = s.pos_ref;
    A.pos_pref = s.prune_buf > 0.0 ? s.pos_pref : nullptr;
    A.brick_key = s.brick_key;
    A.brick_rank = s.brick_rank;
    A.brick_count = s.brick_count;
    A.has_mesh = s.has_mesh;
    A.rebuild = s.rebuild;
    A.prune = s.prune;
    A.status = s.status;
    A.cell_slot = s.cell_slot;
    A.xq = s.xq;
    return A;
}

static FinishArgs finish_args(const DevState &s)
{
    FinishArgs A;
    A.cell_slot = s.cell_slot;
    A.brick_slot = s.brick_slot;
    A.acc_pp = s.acc_pp;
    A.acc_pm = s.acc_pm;
    A.has_mesh = s.has_mesh;
    A.vel = s.vel;
    A.kin_part = s.kin_part;
    A.status = s.status;
    A.rebuild = s.rebuild;
    A.prune = s.prune_buf > 0.0 ? s.prune : nullptr;
    A.prune_count = s.prune_count;
    A.rep_out = s.rep_out;
    return A;
}

template <typename T> void launch_kick_drift(const DevState &s, cudaStream_t st)
{
    k_kick_drift<T><<<pgrid(s.ntot), 256, 0, st>>>(s.reps, s.prep, s.vel, s.acc, s.ntot, drift_args(s));
}

template <typename T> void launch_rescale_drift(const DevState &s, const int *counters, cudaStream_t st)
{
    k_rescale_drift<T><<<s.nblk, PBLK, 0, st>>>(s.reps, s.nrep, s.nblk, s.vel, s.acc, s.kin_part,
                                                counters + 7, drift_args(s));
}

void launch_set_flags(int *flag, int n, int value, cudaStream_t st)
{
    k_set_flags<<<1, 256, 0, st>>>(flag, n, value);
}

template <typename T>
void launch_kick_finish(const DevState &s, int do_kick, double *ep_out, cudaStream_t st, int *counters)
{
    FinishArgs A = finish_args(s);
    A.counters = counters;
    k_kick_finish<T><<<s.nblk, PBLK, 0, st>>>(s.reps, s.nrep, A, s.acc, do_kick, ep_out);
}

template <typename T> void launch_finish_drift(const DevState &s, const DevState &next, cudaStream_t st)
{
    k_finish_drift<T><<<s.nblk, PBLK, 0, st>>>(s.reps, s.nrep, finish_args(s), drift_args(next));
}

void launch_step_reduce(const DevState &s, int mode, int *counters, double *ring, int ring_cap,
                        cudaStream_t st, int recorded, int snap_interval, int snap_cap,
                        const StepSums &sums)
{
    k_step_reduce<<<s.nrep, SR_THREADS, 0, st>>>(s.reps, s.nrep, s.nblk, s.kin_part, s.rep_out, mode,
                                      counters, ring, ring_cap, recorded, snap_interval, snap_cap,
                                      s.status, sums);
}

void launch_snapshot(const DevState &s, const int *counters, double *snap, int *steps,
                     cudaStream_t st)
{
    k_snapshot<<<pgrid(s.ntot), 256, 0, st>>>(s.pos, s.vel, s.acc, s.ntot, counters, snap, steps);
}

void launch_set_counters(int *counters, int run_step, int ring_pos, int it0, cudaStream_t st)
{
    k_set_counters<<<1, 1, 0, st>>>(counters, run_step, ring_pos, it0);
}

template <typename T>
void launch_combine(const DevState &s, int use_pp, int use_pm, int scale_af, double *out,
                    double *ep_out, cudaStream_t st)
{
    using T4 = typename V4<T>::t;
    k_combine<T><<<pgrid(s.ntot), 256, 0, st>>>(s.reps, s.prep, s.cell_slot, s.brick_slot,
                                                (const T4 *)s.acc_pp, (const T4 *)s.acc_pm,
                                                use_pp, use_pm, scale_af, out, ep_out, s.ntot,
                                                s.status);
}

void launch_scale_vel(const DevState &s, cudaStream_t st)
{
    k_scale_vel<<<pgrid(s.ntot), 256, 0, st>>>(s.reps, s.prep, s.rep_out, s.vel, s.ntot);
}

template <typename T>
void launch_nqt(const DevState &s, const double *pos, const double *qmult, int nq, int consecutive,
                double *part, double *out, const int *counters, int ring_cap, cudaStream_t st)
{
    const size_t smem = (size_t)(PBLK / 32) * nq * 6 * sizeof(double);
    if (consecutive)
        k_nqt_partial<T, true><<<s.nq_nblk, PBLK, smem, st>>>(s.reps, s.nrep, pos, qmult, nq, part);
    else
        k_nqt_partial<T, false><<<s.nq_nblk, PBLK, smem, st>>>(s.reps, s.nrep, pos, qmult, nq, part);
    const dim3 rgrid(s.nrep, (nq * 6 + 31) / 32);
    k_nqt_reduce<<<rgrid, NQR_WARPS * 32, 0, st>>>(s.reps, s.nrep, s.nq_nblk, part, nq, out,
                                                   counters, ring_cap);
}

int nqt_particles_per_block() { return PBLK * NQ_PPT; }

template <typename T> void configure_integrate_kernels(int max_nq)
{
    const int smem = (int)((PBLK / 32) * max_nq * 6 * sizeof(double));
    cudaFuncSetAttribute(k_nqt_partial<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_nqt_partial<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

void launch_gf_opt(double kappa, double alpha, int p, int m_alias, int M, double L, double *G_k,
                   double *a_part, cudaStream_t st)
{
    k_gf_opt<<<gf_opt_blocks(M), GF_THREADS, 0, st>>>(kappa, alpha, p, m_alias, M, L, G_k, a_part);
}

int gf_opt_blocks(int M) { return (int)((gf_triples(M) + GF_TRIPLES - 1) / GF_TRIPLES); }

#define P3M_INST(T)                                                                             \
    template void launch_kick_drift<T>(const DevState &, cudaStream_t);                          \
    template void launch_rescale_drift<T>(const DevState &, const int *, cudaStream_t);          \
    template void launch_kick_finish<T>(const DevState &, int, double *, cudaStream_t, int *);   \
    template void launch_finish_drift<T>(const DevState &, const DevState &, cudaStream_t);      \
    template void launch_nqt<T>(const DevState &, const double *, const double *, int, int,      \
                                double *, double *, const int *, int, cudaStream_t);            \
    template void configure_integrate_kernels<T>(int);                                          \
    template void launch_combine<T>(const DevState &, int, int, int, double *, double *,         \
                                    cudaStream_t);
P3M_INST(float)
P3M_INST(double)

}  // namespace p3m
