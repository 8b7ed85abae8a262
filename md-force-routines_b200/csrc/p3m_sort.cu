// Particle keys and counting sorts (PP cells and mesh bricks).
//
// The PP cell of a particle is floor(x / (L/floor(L/rc))) per axis, the same
// cell grid as yukawa_pp.py:17-28 and :44-52; positions are first folded by
// one box length into [0, L) (a particle at exactly x = L lands in cell 0,
// where the reference would index past its grid). The mesh brick is the
// BRICK^3 block of base indices floor(x/h) (yukawa_pm_ord6.py:17-27), folded
// into [0, M).
//
// The cell sort (the grid of the neighbour-list build, cells >= (rc + skin)/2)
// runs only on rebuild steps, per replica: each replica has its own rebuild
// flag, its cells are scanned within its own particle range, and the cell
// kernels skip the work of replicas whose flag is clear -- so a replica's
// lists, and its rounding, do not depend on the other replicas of a batch. It is deterministic: counts and offsets
// come from integer atomics and a scan; the order inside a cell is then
// fixed by sorting each cell's particle indices ascending (rank sort), so
// every rerun builds the same lists. The brick sort runs every step: the
// drift (or key) pass takes each particle's arrival rank in its brick from
// the atomic that counts it, a scan gives the bricks' first slots, and one
// pass writes every particle's stencil offsets and charge to its slot. The
// order inside a brick is whatever the atomics gave; nothing depends on it
// (the assignment sums integers, the gather works per particle). Against a
// stable sort (chunk histograms, a column scan and a warp per chunk placing
// its particles in index order) that is two kernels and two passes fewer:
// per
// step 14.5 -> 6.4 us of drift and sort kernels for 1e4 particles on 64^3, 43
// -> 14 for 1e5 on 128^3, 153 -> 65 for 1e6 on 256^3.
#include "p3m_kernels.h"

namespace p3m {

template <typename T>
__global__ void k_keys(const RepDev *__restrict__ reps, const int *__restrict__ prep,
                       const double *__restrict__ pos, int ntot, int *__restrict__ cell_key,
                       int *__restrict__ cell_sub, int *__restrict__ cell_count,
                       int *__restrict__ brick_key, int *__restrict__ brick_rank,
                       int *__restrict__ brick_count, int has_mesh, int *status)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ntot; i += gridDim.x * blockDim.x) {
        const RepDev &R = reps[prep[i]];
        int c, b, sub;
        particle_keys(R, pos[3 * i + 0], pos[3 * i + 1], pos[3 * i + 2], has_mesh, &c, &b, status,
                      &sub);
        cell_key[i] = c;
        cell_sub[i] = sub;
        atomicAdd(&cell_count[c], 1);
        if (b >= 0) {
            brick_key[i] = b;
            brick_rank[i] = atomicAdd(&brick_count[b * BRICK_CNT_STRIDE], 1);
        }
    }
}

// Cell keys of a rebuild step (the drift kernel computed the brick keys).
__global__ void k_cell_keys(const RepDev *__restrict__ reps, const int *__restrict__ prep,
                            const double *__restrict__ pos, int ntot, int *__restrict__ cell_key,
                            int *__restrict__ cell_sub, int *__restrict__ cell_count,
                            const int *__restrict__ rebuild, int nrep, int *status)
{
    int any = 0;  // nothing to do on most steps
    for (int r = threadIdx.x; r < nrep; r += blockDim.x) any |= rebuild[r];
    if (!__syncthreads_or(any)) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ntot; i += gridDim.x * blockDim.x) {
        const int r = prep[i];
        if (!rebuild[r]) continue;
        const RepDev &R = reps[r];
        int c, b, sub;
        particle_keys(R, pos[3 * i + 0], pos[3 * i + 1], pos[3 * i + 2], 0, &c, &b, status, &sub);
        cell_key[i] = c;
        cell_sub[i] = sub;
        atomicAdd(&cell_count[c], 1);
    }
}

// Exclusive sum over the block's threads of v; *total: the sum of all. sm: 33
// ints. Ends with a barrier.
__device__ int block_excl_scan(int v, int *total, int *sm)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += t;
    }
    if (lane == 31) sm[w] = x;
    __syncthreads();
    if (w == 0) {
        const int own = lane < nw ? sm[lane] : 0;
        int s = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        sm[lane] = s - own;  // exclusive warp totals
        if (lane == 31) sm[32] = s;
    }
    __syncthreads();
    const int e = sm[w] + x - v;
    *total = sm[32];
    __syncthreads();
    return e;
}

// Exclusive scan of count[0], count[STRIDE], ... (n of them) into start[0..n],
// offset by `base` (single block), zeroing the counts and the scatter cursors
// (may be NULL) for the next use. Four entries per thread and round.
template <int STRIDE>
__device__ void block_scan_array(int *count, int *start, int *cursor, int n, int base, int *sm)
{
    int carry = base;
    for (int b0 = 0; b0 < n; b0 += 4 * blockDim.x) {
        const int i0 = b0 + 4 * threadIdx.x;
        int v[4], sum = 0, total;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = i0 + k < n ? count[(i0 + k) * STRIDE] : 0;
            sum += v[k];
        }
        int e = carry + block_excl_scan(sum, &total, sm);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i0 + k < n) {
                start[i0 + k] = e;
                count[(i0 + k) * STRIDE] = 0;
                if (cursor) cursor[i0 + k] = 0;
            }
            e += v[k];
        }
        carry += total;
    }
    if (threadIdx.x == 0) start[n] = carry;
}

// Block r: replica r's cells, within its own particle range [p_off, p_off + n),
// when its rebuild flag is set. Block 0 also writes the list of the rebuilding
// replicas and their cells.
__global__ void k_scan_cells(const RepDev *__restrict__ reps, int nrep, int *cell_count,
                             int *cell_start, int *cell_cursor, const int *__restrict__ rebuild,
                             int *__restrict__ rb_list)
{
    __shared__ int sm[33];
    if (blockIdx.x == 0) {
        int k = 0, cells = 0;
        for (int r0 = 0; r0 < nrep; r0 += blockDim.x) {
            const int r = r0 + threadIdx.x;
            const bool on = r < nrep && rebuild[r] != 0;
            const int nc = on ? reps[r].nc : 0;
            int nk, ncells;
            const int ek = k + block_excl_scan(on ? 1 : 0, &nk, sm);
            const int ec = cells + block_excl_scan(nc * nc * nc, &ncells, sm);
            if (on) {
                rb_list[1 + ek] = r;
                rb_list[nrep + 1 + ek] = ec;
            }
            k += nk;
            cells += ncells;
        }
        if (threadIdx.x == 0) {
            rb_list[0] = k;
            rb_list[nrep + 1 + k] = cells;
        }
    }
    for (int r = blockIdx.x; r < nrep; r += gridDim.x) {
        if (!rebuild[r]) continue;  // block-uniform
        const RepDev &R = reps[r];
        block_scan_array<1>(cell_count + R.cell_off, cell_start + R.cell_off,
                            cell_cursor + R.cell_off, R.nc * R.nc * R.nc, R.p_off, sm);
    }
}

// Block r: replica r's bricks (all its particles lie in them).
__global__ void k_scan_bricks(const RepDev *__restrict__ reps, int nrep, int *brick_count,
                              int *brick_start)
{
    __shared__ int sm[33];
    for (int r = blockIdx.x; r < nrep; r += gridDim.x) {
        const RepDev &R = reps[r];
        block_scan_array<BRICK_CNT_STRIDE>(brick_count + R.brick_off * BRICK_CNT_STRIDE,
                                           brick_start + R.brick_off, nullptr,
                                           R.nb * R.nb * R.nb, R.p_off, sm);
    }
}

__global__ void k_scatter(const int *__restrict__ cell_key, const int *__restrict__ cell_start,
                          int *cell_cursor, int *__restrict__ cell_tmp, int ntot,
                          const int *__restrict__ prep, const int *__restrict__ rebuild,
                          const int *__restrict__ rb_list)
{
    if (rb_list[0] == 0) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ntot; i += gridDim.x * blockDim.x) {
        if (rebuild[prep[i]]) {
            int c = cell_key[i];
            cell_tmp[cell_start[c] + atomicAdd(&cell_cursor[c], 1)] = i;
        }
    }
}

// One warp per cell of the rebuilding replicas: order the cell's particles by
// (sub-cell Morton code, index) -- z-order inside the cell, so the particles
// of one warp of the PP kernel are neighbours in space and walk their
// (similar) lists in step, reading nearby coordinates -- and write, at their
// new slots, the coordinates of the pair stage and the reference point of the
// skin check.
template <typename T>
__global__ void k_fix_cells(const RepDev *__restrict__ reps, int nrep,
                            const int *__restrict__ cell_start, const int *__restrict__ cell_tmp,
                            const int *__restrict__ cell_sub, const double *__restrict__ pos,
                            int *__restrict__ cell_perm, int *__restrict__ cell_slot,
                            double *__restrict__ pos_ref, typename Coord<T>::Q *__restrict__ xq,
                            const int *__restrict__ rb_list)
{
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const int nrb = rb_list[0];
    if (nrb == 0) return;
    const int *rb_cells = rb_list + nrep + 1;
    auto key = [&](int i) { return ((unsigned long long)cell_sub[i] << 32) | (unsigned)i; };
    for (int item = blockIdx.x * wpb + (threadIdx.x >> 5); item < rb_cells[nrb];
         item += gridDim.x * wpb) {
        const int k = find_rep(item, nrb, [&](int j) { return rb_cells[j]; });
        const int r = rb_list[1 + k];
        const int c = reps[r].cell_off + item - rb_cells[k];
        const double inv_L = reps[r].inv_L;
        const int start = cell_start[c], n = cell_start[c + 1] - start;
        for (int e0 = 0; e0 < n; e0 += 32) {
            int e = e0 + lane;
            int v = (e < n) ? cell_tmp[start + e] : 0;
            const unsigned long long kv = (e < n) ? key(v) : ~0ull;
            // rank = keys below kv: 32 keys loaded per pass, compared by shuffle
            int rank = 0;
            for (int f0 = 0; f0 < n; f0 += 32) {
                const int f = f0 + lane;
                const unsigned long long kf = (f < n) ? key(cell_tmp[start + f]) : ~0ull;
                const int m = min(32, n - f0);
                for (int t = 0; t < m; ++t)
                    rank += (__shfl_sync(0xffffffffu, kf, t) < kv) ? 1 : 0;
            }
            if (e < n) {
                const int s = start + rank;
                const double x = pos[3 * v + 0], y = pos[3 * v + 1], z = pos[3 * v + 2];
                cell_perm[s] = v;
                cell_slot[v] = s;
                pos_ref[3 * v + 0] = x;
                pos_ref[3 * v + 1] = y;
                pos_ref[3 * v + 2] = z;
                xq[s] = quantize<T>(x, y, z, inv_L, r);
            }
        }
    }
}

// ---- brick sort ----------------------------------------------------------

// Base index (unwrapped) and offset along one axis (yukawa_pm_ord6.py:17-27).
__device__ __forceinline__ int base_offset(double p, double h, double &off)
{
    int ix = (int)floor(p / h);
    off = (p - (ix + 0.5) * h) / h;
    return ix;
}

__device__ __forceinline__ int wrapM(int i, int M)
{
    i %= M;
    return i < 0 ? i + M : i;
}

// One thread per particle: its slot in brick order, and there its stencil
// offsets (FP64 arithmetic, stored in the bulk precision), its base inside
// the brick and its charge -- what the assignment and the gather read,
// contiguous per brick and computed once for both. SCAN (replicas of up to
// PLACE_SCAN_MAX bricks): blocks are replica-aligned and every block sums its
// replica's brick counts itself, one kernel less on the mesh branch; the
// replica's first block writes the bricks' first slots for the kernels that
// follow, and its last one to have read the counts zeroes them. For up to 148
// blocks (one per SM: 2e3 particles 44.0 -> 43.0 us a step, 1e4 50.6 -> 50.1);
// with more, the repeated sums cost what the kernel saves (20 x 1e4 particles
// 410 against 402 us a step, 1e5 275.8 / 273.9).
constexpr int PLACE_SCAN_MAX = 512;

template <typename T, bool SCAN>
__global__ void __launch_bounds__(PBLK)
k_brick_place(const RepDev *__restrict__ reps, const int *__restrict__ prep, int nrep, int nblk,
              int ntot, const double *__restrict__ pos,
              const double *__restrict__ charge, const int *__restrict__ brick_key,
              const int *__restrict__ brick_rank, int *__restrict__ brick_count,
              int *__restrict__ brick_start, int *__restrict__ brick_slot,
              typename V4<T>::t *__restrict__ slot_pt, T *__restrict__ slot_q,
              int *__restrict__ place_done)
{
    __shared__ int first[SCAN ? PLACE_SCAN_MAX : 1];
    __shared__ int sm[33];
    __shared__ bool reset;
    const int blk = blockIdx.x;
    int i = blk * PBLK + threadIdx.x, r;
    if constexpr (SCAN) {
        r = find_rep(blk, nrep, [&](int k) { return reps[k].blk_off; });
        i = reps[r].p_off + i - reps[r].blk_off * PBLK;
    } else {
        if (i >= ntot) return;
        r = prep[i];
    }
    const RepDev &R = reps[r];
    const int nb = R.nb, M = R.M;
    const bool have = !SCAN || i < R.p_off + R.n;
    int key = 0, rank = 0;
    double x = 0.0, y = 0.0, z = 0.0, q = 0.0;
    if (have) {
        key = brick_key[i];
        rank = brick_rank[i];
        x = pos[3 * i + 0];
        y = pos[3 * i + 1];
        z = pos[3 * i + 2];
        q = charge[i];
    }
    if constexpr (SCAN) {
        static_assert(PLACE_SCAN_MAX == 2 * PBLK, "two bricks per thread");
        const int nbr = nb * nb * nb;
        int *cnt = brick_count + R.brick_off * BRICK_CNT_STRIDE;
        const int b0 = 2 * threadIdx.x;
        const int v0 = b0 < nbr ? cnt[b0 * BRICK_CNT_STRIDE] : 0;
        const int v1 = b0 + 1 < nbr ? cnt[(b0 + 1) * BRICK_CNT_STRIDE] : 0;
        int total;
        const int e = R.p_off + block_excl_scan(v0 + v1, &total, sm);
        // (every thread has its counts: the scan waited for them)
        const int nblk_r = (r + 1 < nrep ? reps[r + 1].blk_off : nblk) - R.blk_off;
        if (threadIdx.x == 0) {
            __threadfence();
            reset = atomicAdd(&place_done[r], 1) == nblk_r - 1;
        }
        first[b0] = e;
        first[b0 + 1] = e + v0;
        __syncthreads();
        if (blk == R.blk_off) {
            if (b0 < nbr) brick_start[R.brick_off + b0] = e;
            if (b0 + 1 < nbr) brick_start[R.brick_off + b0 + 1] = e + v0;
            if (r + 1 == nrep && threadIdx.x == 0) brick_start[R.brick_off + nbr] = R.p_off + R.n;
        }
        if (reset) {
            if (b0 < nbr) cnt[b0 * BRICK_CNT_STRIDE] = 0;
            if (b0 + 1 < nbr) cnt[(b0 + 1) * BRICK_CNT_STRIDE] = 0;
            if (threadIdx.x == 0) place_done[r] = 0;
        }
    }
    if (!have) return;
    const int local = key - R.brick_off;
    const int slot = (SCAN ? first[local] : brick_start[key]) + rank;
    double ox, oy, oz;
    const int ix = base_offset(x, R.h, ox);
    const int iy = base_offset(y, R.h, oy);
    const int iz = base_offset(z, R.h, oz);
    const int lx = wrapM(ix, M) - (local % nb) * BRICK, ly = wrapM(iy, M) - ((local / nb) % nb) * BRICK,
              lz = wrapM(iz, M) - (local / (nb * nb)) * BRICK;
    // a particle outside [-L, 2L) was filed under brick 0 and flagged; it
    // must not reach outside the tile
    const bool in = (unsigned)lx < (unsigned)BRICK && (unsigned)ly < (unsigned)BRICK &&
                    (unsigned)lz < (unsigned)BRICK;
    typename V4<T>::t v;
    v.x = (T)ox;
    v.y = (T)oy;
    v.z = (T)oz;
    v.w = pack_base<T>(in ? lx | (ly << 4) | (lz << 8) : -1);
    brick_slot[i] = slot;
    slot_pt[slot] = v;
    slot_q[slot] = (T)q;
}

static int grid_for(int n, int threads, int cap = 148 * 16)
{
    int g = (n + threads - 1) / threads;
    if (g < 1) g = 1;
    return g < cap ? g : cap;
}

template <typename T> void launch_keys(const DevState &s, cudaStream_t st)
{
    k_keys<T><<<grid_for(s.ntot, 256), 256, 0, st>>>(s.reps, s.prep, s.pos, s.ntot, s.cell_key,
                                                      s.cell_sub, s.cell_count, s.brick_key,
                                                      s.brick_rank, s.brick_count, s.has_mesh,
                                                      s.status);
}

void launch_cell_keys(const DevState &s, cudaStream_t st)
{
    k_cell_keys<<<grid_for(s.ntot, 256), 256, 0, st>>>(s.reps, s.prep, s.pos, s.ntot, s.cell_key,
                                                       s.cell_sub, s.cell_count, s.rebuild,
                                                       s.nrep, s.status);
}

void launch_scan_cells(const DevState &s, cudaStream_t st)
{
    k_scan_cells<<<s.nrep < 1024 ? s.nrep : 1024, 1024, 0, st>>>(
        s.reps, s.nrep, s.cell_count, s.cell_start, s.cell_cursor, s.rebuild, s.rb_list);
}

void launch_scatter(const DevState &s, cudaStream_t st)
{
    k_scatter<<<grid_for(s.ntot, 256), 256, 0, st>>>(s.cell_key, s.cell_start, s.cell_cursor,
                                                      s.cell_tmp, s.ntot, s.prep, s.rebuild,
                                                      s.rb_list);
}

// The brick sort after the key pass; returns the number of kernels.
template <typename T> int launch_place_bricks(const DevState &s, cudaStream_t st)
{
    const int nb = s.max_mesh / BRICK;
    const bool scan = nb * nb * nb <= PLACE_SCAN_MAX && s.nblk <= 148;
    if (!scan)
        k_scan_bricks<<<s.nrep < 1024 ? s.nrep : 1024, 512, 0, st>>>(s.reps, s.nrep, s.brick_count,
                                                                     s.brick_start);
    auto kern = scan ? k_brick_place<T, true> : k_brick_place<T, false>;
    const int grid = scan ? s.nblk : (s.ntot + PBLK - 1) / PBLK;
    kern<<<grid, PBLK, 0, st>>>(s.reps, s.prep, s.nrep, s.nblk, s.ntot, s.pos, s.charge, s.brick_key, s.brick_rank,
                                  s.brick_count, s.brick_start, s.brick_slot,
                                  (typename V4<T>::t *)s.slot_pt, (T *)s.slot_q, s.place_done);
    return scan ? 1 : 2;
}

template <typename T> void launch_fix_cells(const DevState &s, cudaStream_t st)
{
    const int wpb = 8;
    k_fix_cells<T><<<grid_for(s.ncell, wpb), wpb * 32, 0, st>>>(
        s.reps, s.nrep, s.cell_start, s.cell_tmp, s.cell_sub, s.pos, s.cell_perm, s.cell_slot,
        s.pos_ref, (typename Coord<T>::Q *)s.xq, s.rb_list);
}

template void launch_keys<float>(const DevState &, cudaStream_t);
template void launch_keys<double>(const DevState &, cudaStream_t);
template int launch_place_bricks<float>(const DevState &, cudaStream_t);
template int launch_place_bricks<double>(const DevState &, cudaStream_t);
template void launch_fix_cells<float>(const DevState &, cudaStream_t);
template void launch_fix_cells<double>(const DevState &, cudaStream_t);

}  // namespace p3m
