// Particle-mesh (PM) stages: order-6 charge assignment, 3-D FFT of the
// charge mesh, the influence-function multiply with ik differentiation, three
// inverse FFTs of the field components and the order-6 force gather.
//
// This computes what yukawa_pm_ord6.py:440-484 computes:
//   rho   = charge_assgn_6(pos)                       (:445, :6-95)
//   rho_k = fftshift(fftn(rho)); phi_k = G_k rho_k     (:447-451)
//   U_f   = 1/2 sum |rho_k|^2 G_k / V                  (:453-457)
//   E     = (M^3/V) real(ifftn(ifftshift(-i k phi_k))) (:459-480)
//   acc   = Z field_assgn_6(E, pos)                    (:482, :213-312)
// on half spectra (R2C / C2R). Two facts make that equal to the reference's
// full complex transforms: the real part of ifftn equals the C2R transform of
// the Hermitian part of the spectrum, and the -i k_a multiplier of field
// component a is anti-Hermitian on a's own Nyquist plane, where the
// reference's real() therefore cancels it -- so it is zeroed there. U_f sums
// the half spectrum with weight 2 off the kx = 0 and kx = M/2 planes.
//
// Layouts (per replica, concatenated over replicas):
//   tiles   T     [brick][TILE^3]   partial charge of each brick's particles
//   spec    C2<T> [kx][z][y]        kx in [0, M/2], y fastest
//   ek      C2<T> [3][kx][z][y]     field spectra
//   green   T     [kx][z][y]        G_k / V in the same layout
//   efield  T     [3][z][y][x]      real field meshes, x fastest
//
// Assignment is deterministic: each CTA owns one brick of BRICK^3 base
// cells (or a z range of its tile) and adds its particles' 216-node stencils
// into a shared-memory tile of TILE^3 nodes with fixed-point integer atomics,
// whose sums do not depend on the order of the adds (k_assign).
// Overlapping tile halos are summed in a fixed order when the first FFT pass
// reads the mesh.
//
// The FFTs transform lines in two passes of register DFTs (Split) with one
// exchange through shared memory; twiddles come from an FP64-accurate table.
#include "p3m_kernels.h"

namespace p3m {

constexpr int FFT_THREADS = 256;  // a multiple of the largest mesh side (256)

template <typename T> using cplx = typename C2<T>::t;

// signed frequency of index n on an M-point axis
__device__ __forceinline__ int freq(int n, int M) { return n < (M >> 1) ? n : n - M; }

// ---------------------------------------------------------------------------
// FFT lines
// ---------------------------------------------------------------------------

// A line of M = RA RB points is transformed by two passes of register DFTs with
// one exchange through shared memory between them: with n = RB n1 + n2 and
// k = k1 + RA k2,
//   X[k] = sum_n2 W_RB^{n2 k2} [ W_M^{n2 k1} sum_n1 x[n] W_RA^{n1 k1} ],
// pass 1 is an RA-point DFT per n2 (elements RB apart) and the twiddles, pass 2
// an RB-point DFT per k1; both in natural order, no bit reversal. An inverse
// that follows a forward transform starts from what pass 2 left in registers:
// k = k1 + RA k2 over k2 is pass 1 of the swapped split (RB-point DFTs of
// elements RA apart). The lanes of a warp go along the lines where the data is
// already in shared memory (conflict-free) and along the transform where lines
// are contiguous in global memory.
//
// Bound: the x passes by the latency of their tile and spectrum reads, the y
// and z passes by L2 and, at 256^3, HBM (the inverse y pass moves 404 MB in 65
// us, 6.2 TB/s, some four fifths of it HBM's). Radix-2 passes of three stages through shared memory in
// bit-reversed order, which this replaced, moved each element through it eight
// times a line (two now). All passes of a step, before / after, FP32: one 64^3
// mesh 26 / 19 us, 20 of them 125 / 93, 128^3 85 / 54, 256^3 573 / 330; FP64
// one 64^3 38 / 28, 128^3 169 / 95.
template <int LOGM> struct Split {
    static constexpr int RA = fft_ra(LOGM), RB = fft_rb(LOGM);
};

// Twiddle table: for M = 32, 64, 128, 256 the products W_M^{ab} at
// M - 32 + a RB + b (a < RA, b < RB).
template <typename T>
__device__ __forceinline__ void load_twiddles(cplx<T> *tw, const cplx<T> *g)
{
    for (int k = threadIdx.x; k < TWIDDLE_N; k += blockDim.x) tw[k] = g[k];
}

template <typename T> __device__ __forceinline__ cplx<T> cadd(cplx<T> a, cplx<T> b) { return make_c<T>(a.x + b.x, a.y + b.y); }
template <typename T> __device__ __forceinline__ cplx<T> csub(cplx<T> a, cplx<T> b) { return make_c<T>(a.x - b.x, a.y - b.y); }
// times -i (forward) or +i (inverse)
template <typename T, bool INV> __device__ __forceinline__ cplx<T> crot(cplx<T> a)
{
    return INV ? make_c<T>(-a.y, a.x) : make_c<T>(a.y, -a.x);
}
// times w (forward) or conj(w) (inverse)
template <typename T, bool INV> __device__ __forceinline__ cplx<T> ctw(cplx<T> a, cplx<T> w)
{
    if (INV) w.y = -w.y;
    return cmul<T>(a, w);
}

template <typename T, bool INV>
__device__ __forceinline__ void dft4(cplx<T> &a, cplx<T> &b, cplx<T> &c, cplx<T> &d)
{
    const cplx<T> s = cadd<T>(a, c), t = csub<T>(a, c), u = cadd<T>(b, d),
                  v = crot<T, INV>(csub<T>(b, d));
    a = cadd<T>(s, u);
    b = cadd<T>(t, v);
    c = csub<T>(s, u);
    d = csub<T>(t, v);
}

// R-point DFT in registers, natural order in and out, unnormalised
template <typename T, int R, bool INV> __device__ __forceinline__ void dft(cplx<T> (&x)[R])
{
    if constexpr (R == 4) {
        dft4<T, INV>(x[0], x[1], x[2], x[3]);
    } else if constexpr (R == 8) {
        dft4<T, INV>(x[0], x[2], x[4], x[6]);
        dft4<T, INV>(x[1], x[3], x[5], x[7]);
        const T h = (T)0.70710678118654752440L;  // W_8 = (1 -+ i) h
        const cplx<T> o1 = INV ? make_c<T>(h * (x[3].x - x[3].y), h * (x[3].x + x[3].y))
                               : make_c<T>(h * (x[3].x + x[3].y), h * (x[3].y - x[3].x));
        const cplx<T> o2 = crot<T, INV>(x[5]);
        const cplx<T> o3 = INV ? make_c<T>(-h * (x[7].x + x[7].y), h * (x[7].x - x[7].y))
                               : make_c<T>(h * (x[7].y - x[7].x), -h * (x[7].x + x[7].y));
        const cplx<T> e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6], o0 = x[1];
        x[0] = cadd<T>(e0, o0); x[4] = csub<T>(e0, o0);
        x[1] = cadd<T>(e1, o1); x[5] = csub<T>(e1, o1);
        x[2] = cadd<T>(e2, o2); x[6] = csub<T>(e2, o2);
        x[3] = cadd<T>(e3, o3); x[7] = csub<T>(e3, o3);
    } else {
        static_assert(R == 16, "4, 8 or 16 points");
        // 4 x 4: DFTs of elements 4 apart, twiddles W_16^{n2 k1}, DFTs over n2
#pragma unroll
        for (int n = 0; n < 4; ++n) dft4<T, INV>(x[n], x[n + 4], x[n + 8], x[n + 12]);
        const T c1 = (T)0.92387953251128675613L, s1 = (T)0.38268343236508977173L,
                h = (T)0.70710678118654752440L;
        x[5] = ctw<T, INV>(x[5], make_c<T>(c1, -s1));    // W^1
        x[9] = ctw<T, INV>(x[9], make_c<T>(h, -h));      // W^2
        x[13] = ctw<T, INV>(x[13], make_c<T>(s1, -c1));  // W^3
        x[6] = ctw<T, INV>(x[6], make_c<T>(h, -h));      // W^2
        x[10] = crot<T, INV>(x[10]);                     // W^4
        x[14] = ctw<T, INV>(x[14], make_c<T>(-h, -h));   // W^6
        x[7] = ctw<T, INV>(x[7], make_c<T>(s1, -c1));    // W^3
        x[11] = ctw<T, INV>(x[11], make_c<T>(-h, -h));   // W^6
        x[15] = ctw<T, INV>(x[15], make_c<T>(-c1, s1));  // W^9
        // x[4 k1 + n2] now; X[k1 + 4 k2] after the DFT over n2
#pragma unroll
        for (int k = 0; k < 4; ++k) dft4<T, INV>(x[4 * k], x[4 * k + 1], x[4 * k + 2], x[4 * k + 3]);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = a + 1; b < 4; ++b) {
                const cplx<T> t = x[4 * a + b];
                x[4 * a + b] = x[4 * b + a];
                x[4 * b + a] = t;
            }
    }
}

// ---------------------------------------------------------------------------
// Charge assignment
// ---------------------------------------------------------------------------

// Order-6 weights at node offset x (yukawa_pm_ord6.py:29-34), from the even
// and odd parts that mirrored nodes share: w[5 - c](x) = w[c](-x), and the
// outermost are (1 -+ 2x)^5 / 3840. Coefficients are divided by 3840 and 1920
// beforehand (the six divisions per axis were a third of the instructions of
// an FP64 stencil). Multiplications and fused multiply-adds are written out, so
// that every kernel that inlines this rounds alike: a brick's integer sums must
// not depend on which instantiation made them.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

template <typename T>
__device__ __forceinline__ void weights6(T x, T *w)
{
    const T x2 = mul_rn(x, x);
    const T a = fma((T)-2, x, (T)1), b = fma((T)2, x, (T)1);
    const T a2 = mul_rn(a, a), b2 = mul_rn(b, b);
    w[0] = mul_rn(mul_rn(a2, a2), mul_rn(a, (T)(1.0 / 3840)));
    w[5] = mul_rn(mul_rn(b2, b2), mul_rn(b, (T)(1.0 / 3840)));
    const T e1 = fma(x2, fma(x2, (T)(-240.0 / 3840), (T)(840.0 / 3840)), (T)(237.0 / 3840));
    const T o1 = fma(x2, fma(x2, (T)(-160.0 / 3840), (T)(240.0 / 3840)), (T)(750.0 / 3840));
    w[1] = fma(-x, o1, e1);
    w[4] = fma(x, o1, e1);
    const T e2 = fma(x2, fma(x2, (T)(80.0 / 1920), (T)(-440.0 / 1920)), (T)(841.0 / 1920));
    const T o2 = fma(x2, fma(x2, (T)(160.0 / 1920), (T)(-560.0 / 1920)), (T)(770.0 / 1920));
    w[2] = fma(-x, o2, e2);
    w[3] = fma(x, o2, e2);
}

// One CTA of 256 threads per brick, a thread per particle, the 216
// contributions added to a shared tile with integer atomics -- integer sums
// do not depend on the order of the adds, so the result is the same on every
// run, and the brick sort need not order a brick's particles. Each
// contribution q w is scaled by S = 2^k, the largest power of two with
// 0.17 n |q|max S <= 2^B for the brick's n particles (0.17 bounds a product
// of three order-6 weights; |q|max of the replica, in FP64 of the brick), so
// no node sum can exceed 2^B in magnitude. A node is two int32 words:
//
// FP32, B = 22: t = q w S is split exactly into an integer part and an fb-bit
// fraction with the 1.5 * 2^23 rounding constant (exact for |t| < 2^22, no
// float <-> int conversions); the node value is (hi + lo / 2^fb) / S,
// resolved to 2^-fb / S. fb = 16, or fewer for bricks of more than 2^14
// particles, so that the n fractions of a node (each at most 2^fb) cannot
// overflow: n 2^fb <= 2^30.
//
// FP64, B = 62: t rounded to a 64-bit integer, added as its low word and --
// with the carry of that add -- its high word; the number of carries does not
// depend on the order either. Shared memory has no 64-bit add (a
// compare-and-swap loop: 33 us for the 64 bricks of 1e4 particles, against
// 14 with the two words; the ordered FP64 sum it replaced took 34).
// The step 1/S is absolute: 2^-62 of the bound on a node sum, 2^-57 of the
// charge for 156 equal ones, on nodes they hardly reach too (where the weights
// themselves, from offsets that round at 2^-53 of x / h, are no better than some
// 2^-48 of the charge). So that small charges keep theirs beside large ones,
// those of a brick are taken in classes, each within a factor of 2^CLASS_BITS
// of its largest, with a step and a pass over the tile of its own; the classes'
// nodes are added in FP64, the largest first. A brick of one class pays a
// minimum beside its maximum (nothing measurable), every further class its pass:
// 1e4 particles on 64^3 14, 27 and 39 us with one, two and three classes; the
// ordered FP64 sum took 39 on the same box whatever the charges.
//
// Bound: the shared-memory atomics (a warp's add every two cycles; 1280
// bricks of 157 particles 50 -> 42 us without the second pass over positions
// and with shared weight terms, 1e6 particles on 256^3 190 -> 174), in small
// systems as much the CTA's set-up and write-out. With parts > 1, that many
// CTAs share a brick: each owns a z range of the tile's planes, takes the
// particles whose stencils reach it, and writes its planes -- no sums between
// CTAs.
constexpr int A_THREADS = 256;
constexpr int CLASS_BITS = 4;
constexpr float kRound = 12582912.0f;  // 1.5 * 2^23
constexpr int kRoundBits = 0x4B400000;

static size_t assign_smem(int parts)
{
    return (size_t)((TILE + parts - 1) / parts) * TILE * TILE * 2 * sizeof(int);
}

template <typename T, bool SPLIT>
__global__ void __launch_bounds__(A_THREADS)
k_assign(const RepDev *__restrict__ reps, int nrep, const int *__restrict__ brick_start,
         const typename V4<T>::t *__restrict__ slot_pt, const T *__restrict__ slot_q,
         T *__restrict__ tiles, int nbrick, int parts)
{
    extern __shared__ __align__(16) int a_smem[];
    __shared__ int a_src[A_THREADS];  // the chunk's particle slot of each thread, or -1
    __shared__ int a_cnt[32];
    __shared__ double a_qmax[sizeof(T) == 8 ? A_THREADS / 32 : 1];
    const int lane = threadIdx.x & 31;
    const int np_max = SPLIT ? (TILE + parts - 1) / parts : TILE;  // planes of a full part
    int *thi = a_smem, *tlo = a_smem + np_max * TILE * TILE;
    for (int it = blockIdx.x; it < nbrick * (SPLIT ? parts : 1); it += gridDim.x) {
        const int b = SPLIT ? it / parts : it;
        const int z0 = SPLIT ? (it % parts) * np_max : 0;
        const int np = SPLIT ? min(np_max, TILE - z0) : TILE;  // this item's planes z0 .. z0 + np
        if (SPLIT && np <= 0) continue;
        const int nnode = np * TILE * TILE;
        const int r = find_rep(b, nrep, [&](int k) { return reps[k].brick_off; });
        const RepDev &R = reps[r];
        const int local = b - R.brick_off;
        const int p0 = brick_start[b], n = brick_start[b + 1] - p0;
        // classes of charges (FP64): |q| in (low, high], the first without a bound
        double high = 1e308;
        bool more = false, first = true;
        do {
            double qmax = R.qmax, qmin = 1e308, low = 0.0;
            if constexpr (sizeof(T) == 8) {  // the class's largest |q|, and the thread's smallest left
                qmax = 0.0;
                for (int k = threadIdx.x; k < n; k += A_THREADS) {
                    const double q = fabs((double)slot_q[p0 + k]);
                    if (q > high) continue;  // an earlier class's
                    qmax = fmax(qmax, q);
                    if (q > 0.0) qmin = fmin(qmin, q);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) qmax = fmax(qmax, __shfl_xor_sync(0xffffffffu, qmax, o));
                __syncthreads();  // the previous item is done with a_qmax
                if (lane == 0) a_qmax[threadIdx.x >> 5] = qmax;
                __syncthreads();
                for (int k = 0; k < A_THREADS / 32; ++k) qmax = fmax(qmax, a_qmax[k]);
                low = qmax * (1.0 / (1 << CLASS_BITS));
            }
            // S = 2^k with 0.17 n qmax S <= 2^B, k = B - ceil(log2(0.17 n qmax))
            const double bound = fmax(0.17 * (double)(n > 0 ? n : 1) * qmax, 1e-300);
            const long long bits = __double_as_longlong(bound);
            const int ceil2 = (int)(bits >> 52) - 1023 + ((bits & 0xFFFFFFFFFFFFFll) != 0 ? 1 : 0);
            constexpr int B = sizeof(T) == 4 ? 22 : 62, KMAX = sizeof(T) == 4 ? 100 : 1000;
            const int kexp = max(-KMAX, min(B - ceil2, KMAX));
            const double Sd = __longlong_as_double((long long)(kexp + 1023) << 52);
            const T S = (T)Sd;
            const double inv = __longlong_as_double((long long)(1023 - kexp) << 52);  // 1 / S
            const int fb = max(0, min(16, 30 - (32 - __clz(n))));  // n < 2^(32 - clz n)
            const float F = (float)(1 << fb);
            // (the previous pass is done with the tile)
            if constexpr (sizeof(T) == 8) more = __syncthreads_or(qmin <= low);
            else __syncthreads();
            for (int k = threadIdx.x; k < nnode; k += A_THREADS) {
                thi[k] = 0;
                tlo[k] = 0;
            }
            __syncthreads();
            for (int c0 = p0; c0 < p0 + n; c0 += A_THREADS) {
                // The lanes of a warp add at the same offsets from their
                // particles' stencil bases: lanes whose bases share a shared-memory
                // bank conflict on every atomic. The chunk's particles (of those
                // that reach this item's planes) are ranked by bank and dealt
                // round-robin to the warps. Integer sums do not depend on which
                // thread adds what.
                const int c = c0 + threadIdx.x;
                int bank = 0, rank = 0;
                bool use = false;
                if (c < p0 + n) {
                    const int pb = unpack_base(slot_pt[c].w);  // -1: filed under brick 0 and flagged
                    const int lz = (pb >> 8) & 15;
                    use = pb >= 0 && (!SPLIT || (lz + HALO >= z0 && lz < z0 + np));
                    if (sizeof(T) == 8 && (more || !first)) {
                        const double q = fabs((double)slot_q[c]);
                        use = use && q > low && q <= high;
                    }
                    bank = (((lz * TILE + ((pb >> 4) & 15)) * TILE) + (pb & 15)) & 31;
                }
                __syncthreads();  // the previous chunk is done with a_src
                a_src[threadIdx.x] = -1;
                if (threadIdx.x < 32) a_cnt[threadIdx.x] = 0;
                __syncthreads();
                if (use) rank = atomicAdd(&a_cnt[bank], 1);
                const int nch = __syncthreads_count(use);
                if (threadIdx.x < 32) {  // exclusive scan of the bank counts
                    const int v = a_cnt[lane];
                    int x = v;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= o) x += t;
                    }
                    a_cnt[lane] = x - v;
                }
                __syncthreads();
                if (use) {
                    const int q = a_cnt[bank] + rank, nw = (nch + 31) >> 5;
                    a_src[(q % nw) * 32 + q / nw] = c;
                }
                __syncthreads();
                const int p = a_src[threadIdx.x];
                if (p < 0) continue;
                const typename V4<T>::t v = slot_pt[p];
                const int pb = unpack_base(v.w), lz = pb >> 8;
                T wx[6], wy[6], wz[6];
                weights6<T>(v.x, wx);
                weights6<T>(v.y, wy);
                weights6<T>(v.z, wz);
                const T qs = slot_q[p] * S;
                const int base = ((lz - z0) * TILE + ((pb >> 4) & 15)) * TILE + (pb & 15);
#pragma unroll
                for (int g = 0; g < 6; ++g) {
                    if (SPLIT && (unsigned)(lz + g - z0) >= (unsigned)np) continue;
#pragma unroll
                    for (int a = 0; a < 6; ++a) {
                        const T qzy = qs * wz[g] * wy[a];
                        const int row = base + (g * TILE + a) * TILE;
#pragma unroll
                        for (int cx = 0; cx < 6; ++cx) {
                            const T t = mul_rn(qzy, wx[cx]);
                            if constexpr (sizeof(T) == 4) {
                                const float hb = (t - 0.5f) + kRound;    // floor(t), as a float
                                const int hi = __float_as_int(hb) - kRoundBits;
                                const float frac = t - (hb - kRound);      // in [0, 1], exact
                                const int lo = __float_as_int(frac * F + kRound) - kRoundBits;
                                atomicAdd(thi + row + cx, hi);
                                atomicAdd(tlo + row + cx, lo);
                            } else {
                                const long long i = __double2ll_rn(t);
                                const unsigned lo = (unsigned)i;
                                const unsigned old = atomicAdd((unsigned *)tlo + row + cx, lo);
                                atomicAdd(thi + row + cx, (int)(i >> 32) + (old + lo < lo ? 1 : 0));
                            }
                        }
                    }
                }
            }
            __syncthreads();
            T *dst = tiles + R.tile_off + (long long)local * TILE3 + z0 * TILE * TILE;
            // exact as integers, rounded once by the conversion
            const T unit = sizeof(T) == 4 ? (T)(inv / (double)F) : (T)inv;
            for (int k = threadIdx.x; k < nnode; k += A_THREADS) {
                if constexpr (sizeof(T) == 4)
                    dst[k] = (float)(((long long)thi[k] << fb) + tlo[k]) * unit;
                else {
                    const T v = (T)(((long long)thi[k] << 32) | (unsigned)tlo[k]) * unit;
                    dst[k] = first ? v : dst[k] + v;
                }
            }
            high = low;
            first = false;
        } while (more);
    }
}

// A node's charge is the sum of the (up to 8) brick tiles that cover it. Along
// each axis node n lies in the tile of brick n / BRICK at offset n mod BRICK
// and, when that offset is below HALO, also in the halo of the previous
// (periodic) brick's tile at offset + BRICK. A tile element's address is a sum
// of one term per axis, so each axis contributes two candidate offsets.
struct AxisOff {
    int a, b;  // offset in the own brick's tile, in the previous brick's halo
    bool two;  // the halo term exists
};

// sb: elements between consecutive bricks along the axis; st: between
// consecutive tile rows along the axis
__device__ __forceinline__ AxisOff axis_off(int n, int nb, int sb, int st)
{
    const int bk = n / BRICK, o = n - bk * BRICK;
    AxisOff r;
    r.a = bk * sb + o * st;
    r.b = (bk == 0 ? nb - 1 : bk - 1) * sb + (o + BRICK) * st;
    r.two = o < HALO;
    return r;
}
__device__ __forceinline__ AxisOff axis_x(int x, int nb) { return axis_off(x, nb, TILE3, 1); }
__device__ __forceinline__ AxisOff axis_y(int y, int nb) { return axis_off(y, nb, nb * TILE3, TILE); }
__device__ __forceinline__ AxisOff axis_z(int z, int nb)
{
    return axis_off(z, nb, nb * nb * TILE3, TILE * TILE);
}

// The sum over the covering tiles in a fixed order (dz, dy, dx), all loads
// independent; t = the replica's tiles.
template <typename T>
__device__ __forceinline__ T rho_sum(const T *__restrict__ t, const AxisOff &X, const AxisOff &Y,
                                     const AxisOff &Z)
{
    const int zy0 = Z.a + Y.a, zy1 = Z.a + Y.b, zy2 = Z.b + Y.a, zy3 = Z.b + Y.b;
    const bool y1 = Y.two, z1 = Z.two;
    const T v0 = __ldg(t + zy0 + X.a);
    const T v1 = X.two ? __ldg(t + zy0 + X.b) : (T)0;
    const T v2 = y1 ? __ldg(t + zy1 + X.a) : (T)0;
    const T v3 = (y1 && X.two) ? __ldg(t + zy1 + X.b) : (T)0;
    const T v4 = z1 ? __ldg(t + zy2 + X.a) : (T)0;
    const T v5 = (z1 && X.two) ? __ldg(t + zy2 + X.b) : (T)0;
    const T v6 = (z1 && y1) ? __ldg(t + zy3 + X.a) : (T)0;
    const T v7 = (z1 && y1 && X.two) ? __ldg(t + zy3 + X.b) : (T)0;
    return ((v0 + v1) + (v2 + v3)) + ((v4 + v5) + (v6 + v7));
}

// Charge on node (x,y,z) of replica R.
template <typename T>
__device__ __forceinline__ T rho_at(const RepDev &R, const T *__restrict__ tiles, int x, int y, int z)
{
    return rho_sum<T>(tiles + R.tile_off, axis_x(x, R.nb), axis_y(y, R.nb), axis_z(z, R.nb));
}

// ---------------------------------------------------------------------------
// FFT passes
// ---------------------------------------------------------------------------

// Pass A: rows of the charge mesh (reduced from the tiles) -> R2C along x,
// written transposed into spec[kx][z][y]. Item = (replica, z, tile of
// 2 x_lines rows); two real rows share one complex line. Instantiated per mesh
// side. Pass 1 takes its elements straight from the tiles, all of a thread's
// loads independent; pass 2 leaves X[k1 + RA k2] in slot k1 RB + k2 of the
// line, and the two real rows are split from slots k and M - k.
template <int LOGM> __host__ __device__ constexpr int x_stride()
{
    // line stride of the x passes (lines are the fast index): 16 lanes of RB
    // (r2c) or RA (c2r) consecutive transform indices and the lines they span
    // fall on 16 different 8-byte banks
    constexpr int NL = 1 << x_lines_log(LOGM);
    return LOGM == 8 ? NL + 1 : NL + 2;
}

template <typename T, int LOGM>
__device__ __forceinline__ void x_r2c_item(const RepDev &R, int w, const T *__restrict__ tiles,
                                           cplx<T> *__restrict__ spec, cplx<T> *buf,
                                           const cplx<T> *twt)
{
    constexpr int M = 1 << LOGM, RA = Split<LOGM>::RA, RB = Split<LOGM>::RB;
    constexpr int LNL = x_lines_log(LOGM), NL = 1 << LNL, NROW = 2 << LNL;  // complex lines, real rows
    constexpr int NYT = M >> (LNL + 1), NK = (M >> 1) + 1, LS = x_stride<LOGM>();
    const cplx<T> *tw = twt + M - 32;
    const int z = w / NYT, y0 = (w % NYT) * NROW;
    const AxisOff az = axis_z(z, R.nb);
    const T *t = tiles + R.tile_off;
    __syncthreads();
    for (int e = threadIdx.x; e < NL * RB; e += FFT_THREADS) {
        const int n2 = e % RB, l = e / RB;
        const AxisOff ya = axis_y(y0 + 2 * l, R.nb), yb = axis_y(y0 + 2 * l + 1, R.nb);
        cplx<T> x[RA];
#pragma unroll
        for (int n1 = 0; n1 < RA; ++n1) {
            const AxisOff ax = axis_x(RB * n1 + n2, R.nb);
            x[n1].x = rho_sum<T>(t, ax, ya, az);
            x[n1].y = rho_sum<T>(t, ax, yb, az);
        }
        dft<T, RA, false>(x);
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1)
            buf[(k1 * RB + n2) * LS + l] = k1 ? cmul<T>(x[k1], tw[k1 * RB + n2]) : x[0];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < NL * RA; e += FFT_THREADS) {
        const int l = e % NL, k1 = e / NL;
        cplx<T> x[RB];
#pragma unroll
        for (int n2 = 0; n2 < RB; ++n2) x[n2] = buf[(k1 * RB + n2) * LS + l];
        dft<T, RB, false>(x);
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) buf[(k1 * RB + k2) * LS + l] = x[k2];
    }
    __syncthreads();
    // split the two real rows: Xa = (Z[k] + conj Z[M-k])/2, Xb = (Z[k] - conj Z[M-k])/2i
    cplx<T> *out = spec + R.spec_off + (long long)z * M + y0;
    auto slot = [](int k) { return (k % RA) * RB + k / RA; };
    for (int e = threadIdx.x; e < NROW * NK; e += FFT_THREADS) {
        const int j = e & (NROW - 1), k = e >> (LNL + 1);
        const int l = j >> 1;
        const cplx<T> Z = buf[slot(k) * LS + l];
        const cplx<T> Zm = buf[slot((M - k) & (M - 1)) * LS + l];
        cplx<T> X;
        if ((j & 1) == 0) {
            X.x = (T)0.5 * (Z.x + Zm.x);
            X.y = (T)0.5 * (Z.y - Zm.y);
        } else {
            X.x = (T)0.5 * (Z.y + Zm.y);
            X.y = (T)0.5 * (Zm.x - Z.x);
        }
        out[(long long)k * M * M + j] = X;
    }
}

template <typename T>
__global__ void __launch_bounds__(FFT_THREADS, sizeof(T) == 4 ? 3 : 2)
k_fft_x_r2c(const RepDev *__restrict__ reps, int nrep, const T *__restrict__ tiles,
            cplx<T> *__restrict__ spec, const cplx<T> *__restrict__ twg, int nitems)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<T> *tw = reinterpret_cast<cplx<T> *>(smem_raw);
    cplx<T> *buf = tw + TWIDDLE_N;
    load_twiddles<T>(tw, twg);
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int r = find_rep(item, nrep, [&](int k) { return reps[k].wa_off; });
        const RepDev &R = reps[r];
        const int w = item - R.wa_off;
        switch (R.logM) {  // block-uniform: one replica per item
        case 5: x_r2c_item<T, 5>(R, w, tiles, spec, buf, tw); break;
        case 6: x_r2c_item<T, 6>(R, w, tiles, spec, buf, tw); break;
        case 7: x_r2c_item<T, 7>(R, w, tiles, spec, buf, tw); break;
        default: x_r2c_item<T, 8>(R, w, tiles, spec, buf, tw); break;
        }
    }
}

// Passes B / D: FFT along y of contiguous lines spec[kx][z][:], in place. Item
// = (replica, [component,] kx, tile of z lines). `ncomp` arrays of `stride`
// elements are processed (1 forward, 3 inverse). Instantiated per mesh side.
// Pass 1 reads and pass 2 writes global memory directly, lanes along y; the
// strides of the exchange (k1 rows of RB + 1, lines of y_stride) keep both
// sides of it conflict-free.
template <int LOGM> __host__ __device__ constexpr int y_stride()
{
    return LOGM == 8 ? 272 : (LOGM == 7 ? 152 : (LOGM == 6 ? 72 : 40));
}

template <typename T, int LOGM, bool INV>
__device__ __forceinline__ void y_item(const RepDev &R, int w, cplx<T> *__restrict__ data,
                                       long long off, cplx<T> *buf, const cplx<T> *twt)
{
    constexpr int M = 1 << LOGM, RA = Split<LOGM>::RA, RB = Split<LOGM>::RB;
    constexpr int NL = 1 << pencil_log(LOGM), NZT = M / NL, LD = y_stride<LOGM>();
    const cplx<T> *tw = twt + M - 32;
    const int kx = w / NZT, z0 = (w % NZT) * NL;
    cplx<T> *base = data + off + R.spec_off + ((long long)kx * M + z0) * M;
    __syncthreads();
    for (int e = threadIdx.x; e < NL * RB; e += FFT_THREADS) {
        const int n2 = e % RB, l = e / RB;
        cplx<T> x[RA];
#pragma unroll
        for (int n1 = 0; n1 < RA; ++n1) x[n1] = base[l * M + RB * n1 + n2];
        dft<T, RA, INV>(x);
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1)
            buf[l * LD + k1 * (RB + 1) + n2] = k1 ? ctw<T, INV>(x[k1], tw[k1 * RB + n2]) : x[0];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < NL * RA; e += FFT_THREADS) {
        const int k1 = e % RA, l = e / RA;
        cplx<T> x[RB];
#pragma unroll
        for (int n2 = 0; n2 < RB; ++n2) x[n2] = buf[l * LD + k1 * (RB + 1) + n2];
        dft<T, RB, INV>(x);
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) base[l * M + k1 + RA * k2] = x[k2];
    }
}

template <typename T, bool INV>
__global__ void __launch_bounds__(FFT_THREADS)
k_fft_y(const RepDev *__restrict__ reps, int nrep, cplx<T> *__restrict__ data, long long stride,
        int ncomp, const cplx<T> *__restrict__ twg, int nitems_per_comp)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<T> *tw = reinterpret_cast<cplx<T> *>(smem_raw);
    cplx<T> *buf = tw + TWIDDLE_N;
    load_twiddles<T>(tw, twg);
    for (int item = blockIdx.x; item < nitems_per_comp * ncomp; item += gridDim.x) {
        const int comp = item / nitems_per_comp, it = item % nitems_per_comp;
        const int r = find_rep(it, nrep, [&](int k) { return reps[k].wb_off; });
        const RepDev &R = reps[r];
        const int w = it - R.wb_off;
        const long long off = comp * stride;
        switch (R.logM) {  // block-uniform: one replica per item
        case 5: y_item<T, 5, INV>(R, w, data, off, buf, tw); break;
        case 6: y_item<T, 6, INV>(R, w, data, off, buf, tw); break;
        case 7: y_item<T, 7, INV>(R, w, data, off, buf, tw); break;
        default: y_item<T, 8, INV>(R, w, data, off, buf, tw); break;
        }
    }
}

// Pass C: forward FFT along z, U_f partial, phi = (G/V) rho_k, then the three
// field spectra with their inverse z transforms. E_z = IFFT_z(-i kz phi);
// E_x and E_y use psi = IFFT_z(phi) since their multipliers are constant
// along z: E_x = -i kx psi, E_y = -i ky psi. Item = (replica, kx, tile of y);
// instantiated per mesh side. Lanes go along y throughout. The multiplication
// by G and by -i kz happens in registers between the forward transform's pass 2
// and the inverse's pass 1 (split swapped): two exchanges in all.
template <typename T, int LOGM>
__device__ __forceinline__ void z_green_item(const RepDev &R, int w,
                                             const cplx<T> *__restrict__ spec,
                                             const T *__restrict__ green,
                                             cplx<T> *__restrict__ ek, long long nspec,
                                             double *__restrict__ u_out, cplx<T> *buf,
                                             const cplx<T> *twt, double *red)
{
    constexpr int M = 1 << LOGM, RA = Split<LOGM>::RA, RB = Split<LOGM>::RB;
    constexpr int NL = 1 << pencil_log(LOGM), NYT = M / NL;
    const cplx<T> *tw = twt + M - 32;
    cplx<T> *buf2 = buf + M * NL;
    const int kx = w / NYT, y0 = (w % NYT) * NL;
    const long long lbase = R.spec_off + (long long)kx * M * M + y0;  // + z*M + l
    __syncthreads();
    for (int e = threadIdx.x; e < NL * RB; e += FFT_THREADS) {
        const int l = e % NL, n2 = e / NL;
        cplx<T> x[RA];
#pragma unroll
        for (int n1 = 0; n1 < RA; ++n1) x[n1] = spec[lbase + (RB * n1 + n2) * M + l];
        dft<T, RA, false>(x);
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1)
            buf[(k1 * RB + n2) * NL + l] = k1 ? cmul<T>(x[k1], tw[k1 * RB + n2]) : x[0];
    }
    __syncthreads();
    const double wkx = (kx == 0 || kx == (M >> 1)) ? 1.0 : 2.0;
    const T twopi_L = (T)(6.283185307179586477 * R.inv_L);
    double u = 0.0;
    for (int e = threadIdx.x; e < NL * RA; e += FFT_THREADS) {
        const int l = e % NL, k1 = e / NL;
        T g[RB];
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) g[k2] = __ldg(green + lbase + (k1 + RA * k2) * M + l);
        cplx<T> x[RB], f[RB];
#pragma unroll
        for (int n2 = 0; n2 < RB; ++n2) x[n2] = buf[(k1 * RB + n2) * NL + l];
        dft<T, RB, false>(x);
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) {
            const int n = k1 + RA * k2;
            u += wkx * (double)g[k2] * ((double)x[k2].x * x[k2].x + (double)x[k2].y * x[k2].y);
            x[k2] = make_c<T>(g[k2] * x[k2].x, g[k2] * x[k2].y);
            const T kz = (n == (M >> 1)) ? (T)0 : twopi_L * (T)freq(n, M);
            f[k2] = make_c<T>(kz * x[k2].y, -kz * x[k2].x);  // -i kz phi
        }
        dft<T, RB, true>(x);
        dft<T, RB, true>(f);
#pragma unroll
        for (int j = 0; j < RB; ++j) {
            const cplx<T> wj = tw[k1 * RB + j];
            buf[(k1 * RB + j) * NL + l] = ctw<T, true>(f[j], wj);
            buf2[(k1 * RB + j) * NL + l] = ctw<T, true>(x[j], wj);
        }
    }
    __syncthreads();
    const T kxv = (kx == (M >> 1)) ? (T)0 : twopi_L * (T)kx;
    for (int e = threadIdx.x; e < NL * RB; e += FFT_THREADS) {
        const int l = e % NL, j = e / NL;
        const int yy = y0 + l;
        const T kyv = (yy == (M >> 1)) ? (T)0 : twopi_L * (T)freq(yy, M);
        cplx<T> x[RA];
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1) x[k1] = buf[(k1 * RB + j) * NL + l];
        dft<T, RA, true>(x);
#pragma unroll
        for (int i = 0; i < RA; ++i) ek[2 * nspec + lbase + (j + RB * i) * M + l] = x[i];
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1) x[k1] = buf2[(k1 * RB + j) * NL + l];
        dft<T, RA, true>(x);
#pragma unroll
        for (int i = 0; i < RA; ++i) {
            const long long o = lbase + (j + RB * i) * M + l;
            ek[o] = make_c<T>(kxv * x[i].y, -kxv * x[i].x);
            ek[nspec + o] = make_c<T>(kyv * x[i].y, -kyv * x[i].x);
        }
    }
    const double ut = block_sum(u, red);
    if (threadIdx.x == 0) *u_out = ut;
}

template <typename T>
__global__ void __launch_bounds__(FFT_THREADS, sizeof(T) == 4 ? 2 : 1)
k_fft_z_green(const RepDev *__restrict__ reps, int nrep, const cplx<T> *__restrict__ spec,
              const T *__restrict__ green, cplx<T> *__restrict__ ek, long long nspec,
              double *__restrict__ u_part, const cplx<T> *__restrict__ twg, int nitems)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<T> *tw = reinterpret_cast<cplx<T> *>(smem_raw);
    __shared__ double red[32];
    load_twiddles<T>(tw, twg);
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int r = find_rep(item, nrep, [&](int k) { return reps[k].wc_off; });
        const RepDev &R = reps[r];
        const int w = item - R.wc_off;
        cplx<T> *buf = tw + TWIDDLE_N;
        double *u_out = u_part + item;
        switch (R.logM) {  // block-uniform: one replica per item
        case 5: z_green_item<T, 5>(R, w, spec, green, ek, nspec, u_out, buf, tw, red); break;
        case 6: z_green_item<T, 6>(R, w, spec, green, ek, nspec, u_out, buf, tw, red); break;
        case 7: z_green_item<T, 7>(R, w, spec, green, ek, nspec, u_out, buf, tw, red); break;
        default: z_green_item<T, 8>(R, w, spec, green, ek, nspec, u_out, buf, tw, red); break;
        }
    }
}

// Passes B-D fused for meshes whose kx planes fit in shared memory
// (M <= PLANE_MAX): one CTA per (replica, kx) transforms the plane rho_k(kx,z,y)
// along y and z, forms the U_f partial and phi = (G/V) rho_k, and transforms
// back: E_z = IFFT_y IFFT_z(-i kz phi), E_y = IFFT_y(-i ky IFFT_z(phi)), E_x =
// -i kx IFFT_y IFFT_z(phi). One plane read and three plane writes; in between
// the plane goes through shared memory nine times, in eight phases, every pass
// in place (a thread writes the slots it read): after the forward y transform
// column s holds ky = s / RB + RA (s mod RB), which the inverse y transform,
// with the split swapped, takes as it is. The multiplications happen in
// registers between passes. Rows are M + 1 apart: lanes along z or along a row
// fall on different banks; where lanes go along y to meet global memory, the
// rows of a half warp are plane_row()'s, spaced to do the same.
// The energy is summed by 32 consecutive tasks and then over those sums, the same
// tree for either block size: a replica's energy does not depend on whether its
// batch's planes share SMs (tests/test_gpu_batch_planes.py holds that for the
// fields too).
constexpr int PLANE_MAX = 64;

__device__ __forceinline__ int plane_row(int g) { return ((g & 1) << 3) | ((g >> 1) & 7) | (g & ~15); }

template <typename T, int LOGM, int NT>
__device__ __forceinline__ void plane_item(const RepDev &R, int kx, const cplx<T> *__restrict__ spec,
                                           const T *__restrict__ green, cplx<T> *__restrict__ ek,
                                           long long nspec, double *__restrict__ u_out,
                                           cplx<T> *A, cplx<T> *B, const cplx<T> *twt,
                                           double *red)
{
    constexpr int M = 1 << LOGM, RA = Split<LOGM>::RA, RB = Split<LOGM>::RB, LD = M + 1;
    const cplx<T> *tw = twt + M - 32;
    const long long lbase = R.spec_off + (long long)kx * M * M;
    __syncthreads();
    // y, pass 1
    for (int e = threadIdx.x; e < M * RB; e += NT) {
        const int n2 = e % RB, z = plane_row(e / RB);
        cplx<T> x[RA];
#pragma unroll
        for (int n1 = 0; n1 < RA; ++n1) x[n1] = spec[lbase + z * M + RB * n1 + n2];
        dft<T, RA, false>(x);
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1)
            A[z * LD + k1 * RB + n2] = k1 ? cmul<T>(x[k1], tw[k1 * RB + n2]) : x[0];
    }
    __syncthreads();
    // y, pass 2: column k1 RB + k2 = ky k1 + RA k2
    for (int e = threadIdx.x; e < M * RA; e += NT) {
        const int z = e % M, k1 = e / M;
        cplx<T> x[RB];
#pragma unroll
        for (int n2 = 0; n2 < RB; ++n2) x[n2] = A[z * LD + k1 * RB + n2];
        dft<T, RB, false>(x);
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) A[z * LD + k1 * RB + k2] = x[k2];
    }
    __syncthreads();
    // z, pass 1
    for (int e = threadIdx.x; e < M * RB; e += NT) {
        const int s = e % M, n2 = e / M;
        cplx<T> x[RA];
#pragma unroll
        for (int n1 = 0; n1 < RA; ++n1) x[n1] = A[(RB * n1 + n2) * LD + s];
        dft<T, RA, false>(x);
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1)
            A[(RB * k1 + n2) * LD + s] = k1 ? cmul<T>(x[k1], tw[k1 * RB + n2]) : x[0];
    }
    __syncthreads();
    // z, pass 2; U_f, phi, -i kz phi; their inverse z transforms, pass 1
    const double wkx = (kx == 0 || kx == (M >> 1)) ? 1.0 : 2.0;
    const T twopi_L = (T)(6.283185307179586477 * R.inv_L);
    for (int e = threadIdx.x; e < M * RA; e += NT) {
        const int s = e % M, k1 = e / M, y = s / RB + RA * (s % RB);
        T g[RB];
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) g[k2] = __ldg(green + lbase + (k1 + RA * k2) * M + y);
        cplx<T> x[RB], f[RB];
        double u = 0.0;
#pragma unroll
        for (int n2 = 0; n2 < RB; ++n2) x[n2] = A[(k1 * RB + n2) * LD + s];
        dft<T, RB, false>(x);
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) {
            const int n = k1 + RA * k2;
            const double xr = (double)x[k2].x, xi = (double)x[k2].y;
            u = fma(wkx * (double)g[k2], fma(xr, xr, mul_rn(xi, xi)), u);
            x[k2] = make_c<T>(g[k2] * x[k2].x, g[k2] * x[k2].y);
            const T kz = (n == (M >> 1)) ? (T)0 : twopi_L * (T)freq(n, M);
            f[k2] = make_c<T>(kz * x[k2].y, -kz * x[k2].x);  // -i kz phi
        }
        u = warp_sum(u);  // of 32 consecutive e
        if ((threadIdx.x & 31) == 0) red[e >> 5] = u;
        dft<T, RB, true>(x);
        dft<T, RB, true>(f);
#pragma unroll
        for (int j = 0; j < RB; ++j) {
            const cplx<T> wj = tw[k1 * RB + j];
            A[(k1 * RB + j) * LD + s] = ctw<T, true>(f[j], wj);
            B[(k1 * RB + j) * LD + s] = ctw<T, true>(x[j], wj);
        }
    }
    __syncthreads();
    // inverse z, pass 2: rows in natural z
    for (int e = threadIdx.x; e < M * RB; e += NT) {
        const int s = e % M, j = e / M;
        cplx<T> x[RA];
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1) x[k1] = A[(k1 * RB + j) * LD + s];
        dft<T, RA, true>(x);
#pragma unroll
        for (int i = 0; i < RA; ++i) A[(i * RB + j) * LD + s] = x[i];
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1) x[k1] = B[(k1 * RB + j) * LD + s];
        dft<T, RA, true>(x);
#pragma unroll
        for (int i = 0; i < RA; ++i) B[(i * RB + j) * LD + s] = x[i];
    }
    __syncthreads();
    // inverse y, pass 1, of E_z (A) and psi (B); that of -i ky psi waits in
    // registers for A
    constexpr int TPT = (M * RA + NT - 1) / NT;
    cplx<T> h[TPT][RB];
#pragma unroll
    for (int q = 0; q < TPT; ++q) {
        const int e = threadIdx.x + q * NT;
        if (TPT * NT != M * RA && e >= M * RA) break;
        const int z = e % M, k1 = e / M;
        cplx<T> x[RB];
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) x[k2] = A[z * LD + k1 * RB + k2];
        dft<T, RB, true>(x);
#pragma unroll
        for (int j = 0; j < RB; ++j) A[z * LD + k1 * RB + j] = ctw<T, true>(x[j], tw[k1 * RB + j]);
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) {
            const int y = k1 + RA * k2;
            x[k2] = B[z * LD + k1 * RB + k2];
            const T ky = (y == (M >> 1)) ? (T)0 : twopi_L * (T)freq(y, M);
            h[q][k2] = make_c<T>(ky * x[k2].y, -ky * x[k2].x);  // -i ky psi
        }
        dft<T, RB, true>(x);
        dft<T, RB, true>(h[q]);
#pragma unroll
        for (int j = 0; j < RB; ++j) {
            const cplx<T> wj = tw[k1 * RB + j];
            B[z * LD + k1 * RB + j] = ctw<T, true>(x[j], wj);
            h[q][j] = ctw<T, true>(h[q][j], wj);
        }
    }
    __syncthreads();
    // inverse y, pass 2, to global memory: E_z and E_x, then E_y
    const T kxv = (kx == (M >> 1)) ? (T)0 : twopi_L * (T)kx;
    for (int e = threadIdx.x; e < M * RB; e += NT) {
        const int j = e % RB, z = plane_row(e / RB);
        cplx<T> x[RA];
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1) x[k1] = A[z * LD + k1 * RB + j];
        dft<T, RA, true>(x);
#pragma unroll
        for (int i = 0; i < RA; ++i) ek[2 * nspec + lbase + z * M + j + RB * i] = x[i];
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1) x[k1] = B[z * LD + k1 * RB + j];
        dft<T, RA, true>(x);
#pragma unroll
        for (int i = 0; i < RA; ++i)
            ek[lbase + z * M + j + RB * i] = make_c<T>(kxv * x[i].y, -kxv * x[i].x);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < TPT; ++q) {
        const int e = threadIdx.x + q * NT;
        if (TPT * NT != M * RA && e >= M * RA) break;
        const int z = e % M, k1 = e / M;
#pragma unroll
        for (int j = 0; j < RB; ++j) A[z * LD + k1 * RB + j] = h[q][j];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < M * RB; e += NT) {
        const int j = e % RB, z = plane_row(e / RB);
        cplx<T> x[RA];
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1) x[k1] = A[z * LD + k1 * RB + j];
        dft<T, RA, true>(x);
#pragma unroll
        for (int i = 0; i < RA; ++i) ek[nspec + lbase + z * M + j + RB * i] = x[i];
    }
    if (threadIdx.x < 32) {
        static_assert(M * RA <= 32 * 32, "one lane per sum");
        const double ut = warp_sum(threadIdx.x < M * RA / 32 ? red[threadIdx.x] : 0.0);
        if (threadIdx.x == 0) *u_out = ut;
    }
}

template <typename T, int NT>
__global__ void __launch_bounds__(NT, NT == 256 ? 3 : 1)
k_fft_plane(const RepDev *__restrict__ reps, int nrep, const cplx<T> *__restrict__ spec,
            const T *__restrict__ green, cplx<T> *__restrict__ ek, long long nspec,
            double *__restrict__ u_part, const cplx<T> *__restrict__ twg, int nitems)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<T> *tw = reinterpret_cast<cplx<T> *>(smem_raw);
    __shared__ double red[32];
    load_twiddles<T>(tw, twg);
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int r = find_rep(item, nrep, [&](int k) { return reps[k].wp_off; });
        const RepDev &R = reps[r];
        const int kx = item - R.wp_off;
        cplx<T> *A = tw + TWIDDLE_N;
        cplx<T> *B = A + R.M * (R.M + 1);
        if (R.logM == 5)
            plane_item<T, 5, NT>(R, kx, spec, green, ek, nspec, u_part + item, A, B, tw, red);
        else
            plane_item<T, 6, NT>(R, kx, spec, green, ek, nspec, u_part + item, A, B, tw, red);
    }
}

// Pass E: C2R along x of the three field spectra, written as real meshes
// efield[c][z][y][x]. Item = (replica, component, z, tile of 2 x_lines rows); rows
// 2l and 2l+1 share complex line l: Z[k] = Xa[k] + i Xb[k] over the
// Hermitian extension, with the imaginary parts at k = 0 and M/2 dropped.
// Instantiated per mesh side like pass A. Pass 1 takes its elements straight
// from the spectra (k and M - k from the same one: its second read hits L1),
// pass 2 writes the meshes.
template <typename T, int LOGM>
__device__ __forceinline__ void x_c2r_item(const RepDev &R, int comp, int w,
                                           const cplx<T> *__restrict__ ek, long long nspec,
                                           T *__restrict__ efield, long long nmesh, cplx<T> *buf,
                                           const cplx<T> *twt)
{
    constexpr int M = 1 << LOGM, RA = Split<LOGM>::RA, RB = Split<LOGM>::RB;
    constexpr int LNL = x_lines_log(LOGM), NL = 1 << LNL, NROW = 2 << LNL;  // complex lines, real rows
    constexpr int NYT = M >> (LNL + 1);
    // 16 lanes: RA values of k1 on 16 / RA lines
    constexpr int LS = NL + 16 / RA;
    const cplx<T> *tw = twt + M - 32;
    const int z = w / NYT, y0 = (w % NYT) * NROW;
    const cplx<T> *src = ek + comp * nspec + R.spec_off + (long long)z * M + y0;
    __syncthreads();
    for (int e = threadIdx.x; e < NL * RB; e += FFT_THREADS) {
        const int l = e % NL, n2 = e / NL;
        cplx<T> x[RA];
#pragma unroll
        for (int n1 = 0; n1 < RA; ++n1) {
            const int k = RB * n1 + n2, kk = k <= (M >> 1) ? k : M - k;
            const long long o = (long long)kk * M * M + 2 * l;
            cplx<T> a, b;
            if constexpr (sizeof(T) == 4) {  // o is even: one 16-byte load
                const float4 ab = *reinterpret_cast<const float4 *>(src + o);
                a = make_c<T>(ab.x, ab.y);
                b = make_c<T>(ab.z, ab.w);
            } else {
                a = src[o];
                b = src[o + 1];
            }
            if (k == 0 || k == (M >> 1)) x[n1] = make_c<T>(a.x, b.x);
            else if (k < (M >> 1)) x[n1] = make_c<T>(a.x - b.y, a.y + b.x);
            else x[n1] = make_c<T>(a.x + b.y, b.x - a.y);
        }
        dft<T, RA, true>(x);
#pragma unroll
        for (int k1 = 0; k1 < RA; ++k1)
            buf[(n2 * RA + k1) * LS + l] = k1 ? ctw<T, true>(x[k1], tw[k1 * RB + n2]) : x[0];
    }
    __syncthreads();
    T *dst = efield + comp * nmesh + R.mesh_off + ((long long)z * M + y0) * M;
    for (int e = threadIdx.x; e < NL * RA; e += FFT_THREADS) {
        const int k1 = e % RA, l = e / RA;
        cplx<T> x[RB];
#pragma unroll
        for (int n2 = 0; n2 < RB; ++n2) x[n2] = buf[(n2 * RA + k1) * LS + l];
        dft<T, RB, true>(x);
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) {
            dst[2 * l * M + k1 + RA * k2] = x[k2].x;
            dst[(2 * l + 1) * M + k1 + RA * k2] = x[k2].y;
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(FFT_THREADS, sizeof(T) == 4 ? 4 : 2)
k_fft_x_c2r(const RepDev *__restrict__ reps, int nrep, const cplx<T> *__restrict__ ek,
            long long nspec, T *__restrict__ efield, long long nmesh,
            const cplx<T> *__restrict__ twg, int nitems_per_comp)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<T> *tw = reinterpret_cast<cplx<T> *>(smem_raw);
    cplx<T> *buf = tw + TWIDDLE_N;
    load_twiddles<T>(tw, twg);
    for (int item = blockIdx.x; item < nitems_per_comp * 3; item += gridDim.x) {
        const int comp = item / nitems_per_comp, it = item % nitems_per_comp;
        const int r = find_rep(it, nrep, [&](int k) { return reps[k].wa_off; });
        const RepDev &R = reps[r];
        const int w = it - R.wa_off;
        switch (R.logM) {  // block-uniform: one replica per item
        case 5: x_c2r_item<T, 5>(R, comp, w, ek, nspec, efield, nmesh, buf, tw); break;
        case 6: x_c2r_item<T, 6>(R, comp, w, ek, nspec, efield, nmesh, buf, tw); break;
        case 7: x_c2r_item<T, 7>(R, comp, w, ek, nspec, efield, nmesh, buf, tw); break;
        default: x_c2r_item<T, 8>(R, comp, w, ek, nspec, efield, nmesh, buf, tw); break;
        }
    }
}

// ---------------------------------------------------------------------------
// Gather
// ---------------------------------------------------------------------------

// Field at each particle (yukawa_pm_ord6.py:298-300): E = sum over the 216
// stencil nodes of E[node] wz wy wx, written as (Ex, Ey, Ez, Z) in
// brick-sorted order so the caller forms acc = Z E (:308-310). One CTA per
// brick: each field component's TILE^3 neighbourhood of the brick is staged
// in shared memory (coalesced rows), and every particle of the brick reads
// its 216 nodes from there.
//
// Bound: shared-memory reads, 648 words a particle at about two cycles per
// warp's read: a brick's bank counts scatter about their mean, so however the
// particles are dealt, most warps hold two of some bank (1e6 particles on
// 256^3: 144 us of reads in a 200 us kernel).
constexpr int G_THREADS = 256;

// Gather tiles keep rows of GTX nodes (TILE padded up) so each row is filled
// with 16-byte copies: a brick starts on a multiple of 16 nodes and M is a
// multiple of 16, so every 16-byte chunk -- wrapped ones included -- is
// aligned in global and shared memory.
constexpr int GTX = 24;
constexpr int GTILE = TILE * TILE * GTX;

// NB field-tile buffers per CTA: with two, the copy of component c+1 is in
// flight while component c is summed; with one, the CTA is half the size and,
// held to 48 registers, five of them share an SM (FP32: 57 against 63 us on
// the 20 x 64^3 ensemble, with four). The choice is the context's gather_mode.
// The first copies start before the particles are ranked, and a tile stays for
// all chunks of its brick (us a step: FP64 1e4 particles 75.5 -> 73.9, 2e3
// 42.5 -> 42.1; with the fifth CTA 20 x 1e4 404.7 -> 403.3, the mixed batch of
// twelve 636 -> 633).
//
// NC field components per CTA: 3 (a CTA per brick), or 1 (a CTA per brick and
// component: three times the work items, each staging one tile and repeating
// the weights, so the SMs' last wave is shorter and no CTA waits for its own
// next copy).
// gather_mode 1 takes NC = 1 up to GATHER_SPLIT_MAX bricks (measured, us alone
// / step with a CTA per brick against three: 8 bricks 16.5 / 51.8 - 8.3 /
// 46.5, 64 bricks 12.4 / 66.1 - 8.3 / 62.8, FP64 18.5 / 93.1 - 12.4 / 87.5,
// 512 bricks 28.8 / 310.0 - 26.7 / 308.3) and NC = 3 beyond (step, medians of
// six runs from one state: 1280 bricks 395.9 - 396.0, 2048 603.8 - 610, 4096
// 1711 - 1729; an autotuner run, which compares single timings, may pick either
// up to 2048).
constexpr int GATHER_SPLIT_MAX = 512;

template <typename T, int NB, int NC>
__global__ void __launch_bounds__(G_THREADS, sizeof(T) == 4 ? (NB == 1 ? 5 : 1) : 2)
k_gather(const RepDev *__restrict__ reps, int nrep, const int *__restrict__ brick_start,
         const typename V4<T>::t *__restrict__ slot_pt, const T *__restrict__ slot_q,
         const T *__restrict__ efield, long long nmesh,
         typename V4<T>::t *__restrict__ acc_pm, int nbrick)
{
    extern __shared__ __align__(16) unsigned char g_smem[];
    T *tile = reinterpret_cast<T *>(g_smem);
    __shared__ int g_src[G_THREADS];  // per thread of the chunk: its particle's slot, or -1
    __shared__ int g_cnt[32];
    const int lane = threadIdx.x & 31;
    static_assert(NC == 3 || NC == 1, "a whole brick or one component per CTA");
    constexpr int IPB = 3 / NC;  // work items per brick
    for (int it = blockIdx.x; it < nbrick * IPB; it += gridDim.x) {
        const int b = it / IPB, cfirst = (it % IPB) * NC, cend = cfirst + NC;
        const int r = find_rep(b, nrep, [&](int k) { return reps[k].brick_off; });
        const RepDev &R = reps[r];
        const int nb = R.nb, M = R.M, local = b - R.brick_off;
        const int bx = (local % nb) * BRICK, by = ((local / nb) % nb) * BRICK,
                  bz = (local / (nb * nb)) * BRICK;
        const int p0 = brick_start[b], p1 = brick_start[b + 1];
        if (p0 == p1) continue;
        // component tiles through the NB buffers
        auto issue = [&](int comp) {
            constexpr int EPC = 16 / sizeof(T);   // elements per 16-byte chunk
            constexpr int CPR = GTX / EPC;        // chunks per tile row
            constexpr int RP = G_THREADS / CPR;   // tile rows per pass
            static_assert(RP % TILE == 0, "a thread keeps its row's y");
            if (threadIdx.x < RP * CPR) {
                // thread: chunk ch of rows r0, r0 + RP, ... -- fixed x and
                // y, z advancing by RP / TILE
                const int ch = threadIdx.x % CPR, r0 = threadIdx.x / CPR;
                const int gx = (bx + ch * EPC) & (M - 1), gy = (by + r0 % TILE) & (M - 1);
                const T *exy = efield + comp * nmesh + R.mesh_off + (long long)gy * M + gx;
                T *d = tile + (comp % NB) * GTILE + r0 * GTX + ch * EPC;
                for (int tz = r0 / TILE; tz < TILE; tz += RP / TILE, d += RP * GTX)
                    cp_async16(d, exy + (long long)((bz + tz) & (M - 1)) * M * M);
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        __syncthreads();  // the previous brick is done with the buffers
        issue(cfirst);
        if (NB == 2 && cfirst + 1 < cend) issue(cfirst + 1);
        // Up to G_THREADS particles keep slot, base and weights over the
        // components; more are taken in chunks from each staged tile.
        const bool one = p1 - p0 <= G_THREADS;
        T wx[6], wy[6], wz[6];
        int p = -1, base = -1;
        for (int comp = cfirst; comp < cend; ++comp) {
            for (int c0 = p0; c0 < p1; c0 += G_THREADS) {
                if (comp == cfirst || !one) {
                    // Lanes of a warp read their particles' stencils at the same
                    // offsets from different bases, so two lanes whose bases share a
                    // shared-memory bank conflict on every read. The chunk's particles
                    // are ranked by bank (base mod 32) and dealt round-robin to the
                    // warps: each warp gets bases spread over the banks. Which thread
                    // handles a particle does not change its sums.
                    const int nch = min(G_THREADS, p1 - c0);
                    int bank = 0, rank = 0;
                    if (threadIdx.x < nch) {
                        const int pb = max(0, unpack_base(slot_pt[c0 + threadIdx.x].w));
                        bank = (((pb >> 8) * TILE + ((pb >> 4) & 15)) * GTX + (pb & 15)) & 31;
                    }
                    __syncthreads();  // the previous chunk / brick is done with g_*
                    g_src[threadIdx.x] = -1;
                    if (threadIdx.x < 32) g_cnt[threadIdx.x] = 0;
                    __syncthreads();
                    if (threadIdx.x < nch) rank = atomicAdd(&g_cnt[bank], 1);
                    __syncthreads();
                    if (threadIdx.x < 32) {  // exclusive scan of the bank counts
                        const int v = g_cnt[lane];
                        int x = v;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const int t = __shfl_up_sync(0xffffffffu, x, o);
                            if (lane >= o) x += t;
                        }
                        g_cnt[lane] = x - v;
                    }
                    __syncthreads();
                    if (threadIdx.x < nch) {
                        const int q = g_cnt[bank] + rank, nw = (nch + 31) >> 5;
                        g_src[(q % nw) * 32 + q / nw] = c0 + threadIdx.x;
                    }
                    __syncthreads();
                    p = g_src[threadIdx.x];
                    base = -1;
                    if (p >= 0) {
                        const typename V4<T>::t v = slot_pt[p];
                        const int pb = unpack_base(v.w);  // -1: flagged by the key pass
                        if (pb >= 0) base = ((pb >> 8) * TILE + ((pb >> 4) & 15)) * GTX + (pb & 15);
                        weights6<T>(v.x, wx);
                        weights6<T>(v.y, wy);
                        weights6<T>(v.z, wz);
                    }
                }
                if (c0 == p0) {
                    if (NB == 2 && comp + 1 < cend) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
                    else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
                    __syncthreads();
                }
                const T *tl = tile + (comp % NB) * GTILE;
                T acc = 0;
                if (base >= 0) {
                    // separable contraction: sum_g wz sum_a wy sum_c wx E
#pragma unroll
                    for (int g = 0; g < 6; ++g) {
                        T sg = 0;
#pragma unroll
                        for (int a = 0; a < 6; ++a) {
                            const T *row = tl + base + (g * TILE + a) * GTX;
                            T sa = 0;
#pragma unroll
                            for (int c = 0; c < 6; ++c) sa += wx[c] * row[c];
                            sg += wy[a] * sa;
                        }
                        acc += wz[g] * sg;
                    }
                }
                if (p >= 0) {
                    T *o = reinterpret_cast<T *>(acc_pm + p);  // (Ex, Ey, Ez, Z)
                    o[comp] = acc;
                    if (comp == 0) o[3] = slot_q[p];
                }
            }
            if (comp + NB < cend) {
                __syncthreads();  // buffer comp % NB is refilled
                issue(comp + NB);
            }
        }
    }
}

// Per-replica U_f = 1/2 sum over the replica's pass-C partials.
__global__ void k_reduce_pm(const RepDev *__restrict__ reps, int nrep,
                            const double *__restrict__ u_part, int wc_total, int wp_total,
                            double *__restrict__ rep_out)
{
    const int lane = threadIdx.x & 31;
    for (int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < nrep;
         r += gridDim.x * (blockDim.x >> 5)) {
        if (reps[r].M == 0) {
            if (lane == 0) rep_out[8 * r + RO_UPM] = 0.0;
            continue;
        }
        // multi-pass items [wc_off, ...) and plane items (stored after wc_total)
        const int b = reps[r].wc_off, e = (r + 1 < nrep) ? reps[r + 1].wc_off : wc_total;
        const int pb = wc_total + reps[r].wp_off,
                  pe = wc_total + ((r + 1 < nrep) ? reps[r + 1].wp_off : wp_total);
        double t = 0.0;
        for (int k = b + lane; k < e; k += 32) t += u_part[k];
        for (int k = pb + lane; k < pe; k += 32) t += u_part[k];
        t = warp_sum(t);
        if (lane == 0) rep_out[8 * r + RO_UPM] = 0.5 * t;
    }
}

// ---------------------------------------------------------------------------
// Conversions used by the compat entry points
// ---------------------------------------------------------------------------

// Influence function from the reference's fftshifted (M,M,M) FP64 layout
// (index n <-> k = 2 pi (n - M/2)/L) into green[kx][z][y] / V.
template <typename T>
__global__ void k_green_from_shifted(const RepDev *__restrict__ reps, int rep,
                                     const double *__restrict__ gk, T *__restrict__ green)
{
    const RepDev &R = reps[rep];
    const int M = R.M, h = M >> 1, nk = h + 1;
    const long long n = (long long)nk * M * M;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        const int y = (int)(e % M), z = (int)((e / M) % M), kx = (int)(e / ((long long)M * M));
        const int sx = (kx + h) & (M - 1), sy = (y + h) & (M - 1), sz = (z + h) & (M - 1);
        green[R.spec_off + e] = (T)(gk[((long long)sz * M + sy) * M + sx] * R.inv_V);
    }
}

template <typename T>
__global__ void k_tiles_to_mesh(const RepDev *__restrict__ reps, int rep,
                                const T *__restrict__ tiles, double *__restrict__ rho)
{
    const RepDev &R = reps[rep];
    const int M = R.M;
    const long long n = (long long)M * M * M;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(e % M), y = (int)((e / M) % M), z = (int)(e / ((long long)M * M));
        rho[e] = (double)rho_at<T>(R, tiles, x, y, z);
    }
}

template <typename T>
__global__ void k_efield_from_mesh(const RepDev *__restrict__ reps, int rep,
                                   const double *__restrict__ ex, const double *__restrict__ ey,
                                   const double *__restrict__ ez, T *__restrict__ efield,
                                   long long nmesh)
{
    const RepDev &R = reps[rep];
    const long long n = (long long)R.M * R.M * R.M;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        efield[R.mesh_off + e] = (T)ex[e];
        efield[nmesh + R.mesh_off + e] = (T)ey[e];
        efield[2 * nmesh + R.mesh_off + e] = (T)ez[e];
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

// shared memory of the passes for meshes up to maxM: the twiddles and the
// largest exchange buffer of the sides up to maxM
template <typename T> static size_t y_smem(int maxM)
{
    const int n = maxM >= 128 ? (32 * y_stride<7>() > 16 * y_stride<8>() ? 32 * y_stride<7>() : 16 * y_stride<8>())
                              : 32 * y_stride<6>();
    return (size_t)(TWIDDLE_N + n) * sizeof(cplx<T>);
}

template <typename T> static size_t z_smem(int maxM)
{
    return (size_t)(TWIDDLE_N + 2 * (maxM >= 128 ? 256 << pencil_log(8) : 64 << pencil_log(6))) * sizeof(cplx<T>);
}
static_assert((128 << pencil_log(7)) <= (256 << pencil_log(8)), "z exchange at 128");

template <typename T> static size_t plane_smem(int M)
{
    return (TWIDDLE_N + 2 * (size_t)M * (M + 1)) * sizeof(cplx<T>);
}

template <typename T> static size_t x_smem(int maxM)
{
    return (size_t)(TWIDDLE_N + (maxM >= 128 ? 256 * x_stride<8>() : 64 * x_stride<6>())) * sizeof(cplx<T>);
}
static_assert(128 * x_stride<7>() <= 256 * x_stride<8>(), "x exchange at 128");

template <typename K> static void set_smem(K kernel, size_t bytes)
{
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

static int grid_items(int n, int cap = 148 * 8) { return n < cap ? (n > 0 ? n : 1) : cap; }

template <typename T> void configure_mesh_kernels()
{
    set_smem(k_assign<T, false>, assign_smem(1));
    set_smem(k_assign<T, true>, assign_smem(1));
    set_smem(k_fft_x_r2c<T>, x_smem<T>(256));
    set_smem(k_fft_y<T, false>, y_smem<T>(256));
    set_smem(k_fft_y<T, true>, y_smem<T>(256));
    set_smem(k_fft_z_green<T>, z_smem<T>(256));
    set_smem(k_fft_x_c2r<T>, x_smem<T>(256));
    set_smem(k_gather<T, 1, 3>, GTILE * sizeof(T));
    set_smem(k_gather<T, 1, 1>, GTILE * sizeof(T));
    if constexpr (sizeof(T) == 4) set_smem(k_gather<T, 2, 3>, 2 * GTILE * sizeof(T));
    if constexpr (sizeof(T) == 4) set_smem(k_fft_plane<T, 256>, plane_smem<T>(PLANE_MAX));
    set_smem(k_fft_plane<T, 512>, plane_smem<T>(PLANE_MAX));
}

// CTAs per brick of the assignment: two for up to 32 bricks (FP32, one
// against two CTAs: 12.4 / 10.3 us at 8 bricks of 250 particles, 12.4 / 11.8
// at 32), one from there on, where the repeated set-up costs as much as the
// halved atomics save (8.3 / 8.3 us at 64 bricks, 9.2 / 10.3 at 128, 22 / 27
// at 512; three or more CTAs nowhere better than two).
int assign_parts_for(int nbrick) { return nbrick <= 32 ? 2 : 1; }

template <typename T> void launch_assign(const DevState &s, cudaStream_t st)
{
    using A = typename V4<T>::t;
    const int parts = s.assign_parts;
    const int grid = grid_items(s.nbrick * parts, 148 * 16);
    auto go = [&](auto kern) {
        kern<<<grid, A_THREADS, assign_smem(parts), st>>>(s.reps, s.nrep, s.brick_start, (const A *)s.slot_pt,
                                                   (const T *)s.slot_q, (T *)s.tiles, s.nbrick, parts);
    };
    if (parts > 1) go(k_assign<T, true>);
    else go(k_assign<T, false>);
}

template <typename T> void launch_fft_forward(const DevState &s, cudaStream_t st)
{
    using C = cplx<T>;
    const int maxM = s.max_mesh;
    k_fft_x_r2c<T><<<grid_items(s.wa), FFT_THREADS, x_smem<T>(maxM), st>>>(s.reps, s.nrep, (const T *)s.tiles,
                                                                (C *)s.spec, (const C *)s.twiddle, s.wa);
    if (s.wb > 0) {
        k_fft_y<T, false><<<grid_items(s.wb), FFT_THREADS, y_smem<T>(maxM), st>>>(
            s.reps, s.nrep, (C *)s.spec, s.nspec, 1, (const C *)s.twiddle, s.wb);
        k_fft_z_green<T><<<grid_items(s.wc), FFT_THREADS, z_smem<T>(maxM), st>>>(
            s.reps, s.nrep, (const C *)s.spec, (const T *)s.green, (C *)s.ek, s.nspec, s.u_pm_part,
            (const C *)s.twiddle, s.wc);
    }
    if (s.wp > 0) {
        // 512 threads a plane where every plane has an SM (FP32 64^3, 512 / 256
        // threads: 33 planes 8.9 / 9.9 us, 132 planes 9.4 / 10.5), and in FP64,
        // whose two planes take an SM's shared memory; 256 where planes share
        // SMs, three CTAs each (264 planes 18.0 / 15.4 us, 660 45.2 / 32.9)
        auto go = [&](auto kern, int nt) {
            kern<<<grid_items(s.wp), nt, plane_smem<T>(s.max_plane), st>>>(
                s.reps, s.nrep, (const C *)s.spec, (const T *)s.green, (C *)s.ek, s.nspec,
                s.u_pm_part + s.wc, (const C *)s.twiddle, s.wp);
        };
        if constexpr (sizeof(T) == 4) {
            if (s.wp > 148) go(k_fft_plane<T, 256>, 256);
            else go(k_fft_plane<T, 512>, 512);
        } else {
            go(k_fft_plane<T, 512>, 512);
        }
    }
}

int fft_kernel_count(const DevState &s) { return 2 + (s.wb > 0 ? 3 : 0) + (s.wp > 0 ? 1 : 0); }
int plane_max_mesh() { return PLANE_MAX; }  // the largest side the plane kernel takes

template <typename T> void launch_fft_inverse(const DevState &s, cudaStream_t st)
{
    using C = cplx<T>;
    if (s.wb > 0)
        k_fft_y<T, true><<<grid_items(3 * s.wb), FFT_THREADS, y_smem<T>(s.max_mesh), st>>>(
            s.reps, s.nrep, (C *)s.ek, s.nspec, 3, (const C *)s.twiddle, s.wb);
    k_fft_x_c2r<T><<<grid_items(3 * s.wa), FFT_THREADS, x_smem<T>(s.max_mesh), st>>>(
        s.reps, s.nrep, (const C *)s.ek, s.nspec, (T *)s.efield, s.nmesh, (const C *)s.twiddle,
        s.wa);
}

template <typename T> void launch_gather(const DevState &s, cudaStream_t st)
{
    using A = typename V4<T>::t;
    if (sizeof(T) == 4 && s.gather_mode == 2)
        k_gather<T, 2, 3><<<grid_items(s.nbrick, 148 * 16), G_THREADS, 2 * GTILE * sizeof(T), st>>>(
            s.reps, s.nrep, s.brick_start, (const A *)s.slot_pt, (const T *)s.slot_q, (const T *)s.efield,
            s.nmesh, (A *)s.acc_pm, s.nbrick);
    else if (s.gather_mode == 0 || s.nbrick <= GATHER_SPLIT_MAX)
        k_gather<T, 1, 1><<<grid_items(3 * s.nbrick, 148 * 16), G_THREADS, GTILE * sizeof(T), st>>>(
            s.reps, s.nrep, s.brick_start, (const A *)s.slot_pt, (const T *)s.slot_q, (const T *)s.efield,
            s.nmesh, (A *)s.acc_pm, s.nbrick);
    else
        k_gather<T, 1, 3><<<grid_items(s.nbrick, 148 * 16), G_THREADS, GTILE * sizeof(T), st>>>(
            s.reps, s.nrep, s.brick_start, (const A *)s.slot_pt, (const T *)s.slot_q, (const T *)s.efield,
            s.nmesh, (A *)s.acc_pm, s.nbrick);
}

void launch_reduce_pm(const DevState &s, cudaStream_t st)
{
    k_reduce_pm<<<(s.nrep + 3) / 4, 128, 0, st>>>(s.reps, s.nrep, s.u_pm_part, s.wc, s.wp,
                                                  s.rep_out);
}

template <typename T>
void launch_green_from_host_layout(const DevState &s, int rep, const double *gk_dev, cudaStream_t st)
{
    k_green_from_shifted<T><<<592, 256, 0, st>>>(s.reps, rep, gk_dev, (T *)s.green);
}

template <typename T> void launch_tiles_to_mesh(const DevState &s, int rep, double *rho, cudaStream_t st)
{
    k_tiles_to_mesh<T><<<592, 256, 0, st>>>(s.reps, rep, (const T *)s.tiles, rho);
}

template <typename T>
void launch_efield_from_mesh(const DevState &s, int rep, const double *ex, const double *ey,
                             const double *ez, cudaStream_t st)
{
    k_efield_from_mesh<T><<<592, 256, 0, st>>>(s.reps, rep, ex, ey, ez, (T *)s.efield, s.nmesh);
}

#define P3M_INST(T)                                                                        \
    template void configure_mesh_kernels<T>();                                              \
    template void launch_assign<T>(const DevState &, cudaStream_t);                         \
    template void launch_fft_forward<T>(const DevState &, cudaStream_t);                    \
    template void launch_fft_inverse<T>(const DevState &, cudaStream_t);                    \
    template void launch_gather<T>(const DevState &, cudaStream_t);                         \
    template void launch_green_from_host_layout<T>(const DevState &, int, const double *,   \
                                                   cudaStream_t);                          \
    template void launch_tiles_to_mesh<T>(const DevState &, int, double *, cudaStream_t);   \
    template void launch_efield_from_mesh<T>(const DevState &, int, const double *,         \
                                             const double *, const double *, cudaStream_t);
P3M_INST(float)
P3M_INST(double)

}  // namespace p3m
