// Compile-time-sized plane pipeline (the fast path of lh_plane.cu).
//
// Every transform is a two-pass register FFT (lh_fft.cuh) whose index
// arithmetic folds to constants; one template per stage, instantiated for
// the Ngal sizes of the usual grids.  One CTA per work item; each lane reads
// its one outer-twiddle base from the table in global memory, so shared
// memory holds only the transform data.
//
// Staging (per instance, inside I.S; the kRoundStreams chunk rounds in
// flight use disjoint shares):
//   Sin  [cap+2*kRoundStreams][3][Mz][nxh]  z-inverse of u1, u3 and u2 on the y rows of
//        a round's planes plus one halo row each side; x stays spectral.
//   Sprod[cap][6][Mz][nxh]    the six products after the forward x
//        transform, one slot per plane of a round.
// The y interpolations of the reference (interp_u/interp_v, FOU3D.f90:
// 373-418) are linear and commute with the z transform, so they are applied
// to the z-transformed rows in the x stage: the z inverse runs on three
// fields per plane instead of six.
#include <algorithm>
#include <cstdlib>

#include "lh_fft.cuh"

// Launch bounds (max threads, min resident CTAs per SM) each kernel's
// register allocation is sized for.
#ifndef LH_ZINV_T
#define LH_ZINV_T 256
#endif
#ifndef LH_ZINV_B
#define LH_ZINV_B 3
#endif
#ifndef LH_ZFWD_T
#define LH_ZFWD_T 256
#endif
#ifndef LH_ZFWD_B
#define LH_ZFWD_B 3
#endif
// The z kernels at the lengths of 18 and more threads per vector hold longer
// register FFTs: at three CTAs per SM (80 registers) they spilled 0.1-0.8 KB per
// thread.  There the bound is LH_LARGE_B CTAs per SM (128 registers, no spills).
// Measured on B200 (ms per RK3 step): 256^2 x 257 12.32 -> 10.15; 192^2 x 257
// 5.04 -> 4.88, x 153 3.11 -> 3.01, x 97 2.00 -> 1.93; at Ngal 192 two CTAs lost
// in the step graph.
#ifndef LH_LARGE_B
#define LH_LARGE_B 2
#endif
#define LH_MINB(N, B) (Plan2<N>::N1 >= 18 || Plan2<N>::N2 >= 18 ? LH_LARGE_B : (B))
#include "lh_kernels.cuh"
#include "lh_xprod.cuh"

namespace lh {

constexpr int kXprodThreads = 128;  // most threads of a k_xprod_r CTA

__device__ __forceinline__ double2 *sin_field(const Inst &I, int p, int f)
{
    return I.S + ((size_t)p * 3 + f) * I.Mz * I.nxh;
}
__device__ __forceinline__ double2 *sprod_slot(const Inst &I, int s)
{
    return I.S + ((size_t)(I.chunk + 2 * kRoundStreams) * 3 + (size_t)s * kNumProducts) * I.Mz * I.nxh;
}

// ---------------------------------------------------------------------------
// z inverse of one (y row jp, field f in {u1, u3, u2}, block of cb x modes):
// the pruned cft of four_to_phys_u (FOU3D.f90:653-679), -> Sin[slot][f]
// Elements from one k1 block of v vectors to the next in the exchange of a two-pass z
// transform: the threads write it in their own order, and the second pass, whose
// neighbouring rows are whole blocks apart, reads on from bank to bank as well.
template <int NZ>
__host__ __device__ constexpr int zblock(int v)
{
    return Plan2<NZ>::N2 * v + ((v * (1 + 7 * Plan2<NZ>::N2)) & 7);
}

template <int NZ>
__global__ void __launch_bounds__(LH_ZINV_T, LH_MINB(NZ, LH_ZINV_B)) k_zinv_f(const Inst *__restrict__ insts, const Work *__restrict__ work,
                                                         int count, int cb)
{
    constexpr int N1 = Plan2<NZ>::N1, N2 = Plan2<NZ>::N2;
    constexpr int Nz = 2 * NZ / 3;
    extern __shared__ double2 sm[];
    double2 *T = sm;
    if ((int)blockIdx.x >= count) return;
    const double2 *tw = insts[work[blockIdx.x].inst].twz;  // depends on Mz only
    const int t = threadIdx.x, v = t % cb, r = t / cb, zb = zblock<NZ>(cb);
    const double2 twr = __ldg(tw + r);  // outer-twiddle base W^r, issued before the data loads
    {
        const Work w = work[blockIdx.x];
        const Inst &I = insts[w.inst];
        const int nxh = I.nxh, nc = I.nc;
        const int nblk = (nxh + cb - 1) / cb;
        const int f = w.blk / nblk, i = (w.blk % nblk) * cb + v;
        const double2 *src = (f == 0 ? I.U1 : (f == 1 ? I.U3 : I.U2)) + (size_t)w.j * nc;
        const bool ok = i < nxh;
        if (r < N2) {
            double2 a[N1];
#pragma unroll
            for (int n1 = 0; n1 < N1; n1++) {
                const int n = r + N2 * n1;
                int kr = -1;
                if (n < Nz / 2) kr = n;
                else if (n >= NZ - Nz / 2) kr = n - (NZ - Nz);
                a[n1] = (kr >= 0 && ok) ? src[kr * nxh + i] : make_double2(0.0, 0.0);
            }
            DFT<N1, +1, NZ>::run(a, tw);
            TwStep ts(twr);
#pragma unroll
            for (int k1 = 0; k1 < N1; k1++) {
                double2 z = a[k1];
                if (k1 > 0) z = twiddle<+1>(ts.next(), z);
                T[k1 * zb + t] = z;
            }
        }
        __syncthreads();
        if (r < N1) {
            double2 b[N2];
#pragma unroll
            for (int n2 = 0; n2 < N2; n2++) b[n2] = T[r * zb + n2 * cb + v];
            DFT<N2, +1, NZ>::run(b, tw);
            if (ok) {
                double2 *dst = sin_field(I, w.slot, f) + i;
#pragma unroll
                for (int k2 = 0; k2 < N2; k2++) dst[(size_t)(r + N1 * k2) * nxh] = b[k2];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// x transforms and products of one (plane j, block of rb z rows): xrow on rows
// gathered from Sin with the y interpolations (interp_v FOU3D.f90:407, interp_u
// :387): u1(j), u3(j); u2 at centre j, u2(j); u1, u3 at face j -> Sprod[slot]
// What bounds it: the FP64 pipe (51 % of its cycles at Mx = 192) and the shared-memory
// / L1 data pipe (50 %), at the warps that 168 registers leave (three CTAs of
// 128).  x products alone, us a substep on B200 at 96 MB of staging: one vector a half
// warp, or block-synchronous where vectors do not fit a warp -> products in registers
// -> tasks packed on consecutive lanes: 64^2 x 153 72 -> 61 -> 57, 128^2 x 153 231 ->
// 188 -> 181, 192^2 x 257 958 -> 910 -> 850, 256^2 x 257 1955 -> 1310 -> 1275; the substep
// 128 -> 114 -> 110, 401 -> 363 -> 357, 1639 -> 1554 -> 1505, 3258 -> 2685 -> 2640.  Before
// the packing, four CTAs an SM (128 registers) spilled: 372 us at 128^2, 1764 at
// 192^2; three instead of two at Mx = 384 3150.  Two at N2 = 18: 192^2 x 257 706 for 641
// (300 MB).
template <int NX>
__global__ void __launch_bounds__(kXprodThreads, XPlan<NX>::N2 <= 6 ? 4 : (XPlan<NX>::N2 <= 18 ? 3 : 2))
    k_xprod_r(const Inst *__restrict__ insts, const Work *__restrict__ work, int rb, int want_max)
{
    using XP = XPlan<NX>;
    using XK = XPack<NX>;
    constexpr int KQ = XP::KQ, nxh = NX / 3 + 1;
    extern __shared__ double2 sm[];
    const Work w = work[blockIdx.x];
    const Inst &I = insts[w.inst];
    const int Mz = I.Mz, j = w.j;
    // first z row of this warp and how many there are; not packed: this lane's row and
    // whether there is one
    const int lane = threadIdx.x & 31;
    const bool on = lane < XP::RW * XP::N1;
    const int row0 = (threadIdx.x >> 5) * XP::RW + (XK::value || !on ? 0 : lane / XP::N1), q0 = w.blk * rb + row0;
    const int left = min(rb - row0, Mz - q0), rows = XK::value ? min(XP::RW, left) : (on && left > 0);
    // this row in the planes the y interpolations read, in field strides from u1(j): u2(j-1)
    // -1, u1(j) 0, u3(j) 1, u2(j) 2, u1(j+1) 3, u3(j+1) 4; 32-bit offsets
    const int fs = Mz * nxh;
    const double2 *const U = sin_field(I, w.aux + 1, 0) + (size_t)min(q0, Mz - 1) * nxh;
    double2 *const S = sprod_slot(I, w.slot) + (size_t)min(q0, Mz - 1) * nxh;
    const double dnv = 1.0 / (I.yv[j] - I.yv[j - 1]), dnu = 1.0 / (I.yu[j + 1] - I.yu[j]);
    const double w0v = (I.yu[j] - I.yv[j - 1]) * dnv, w1v = (I.yv[j] - I.yu[j]) * dnv;
    const double w0u = (I.yv[j] - I.yu[j]) * dnu, w1u = (I.yu[j + 1] - I.yv[j]) * dnu;
    const bool track = want_max && I.dt_mode == 0 && j <= I.nyu - 1;  // maxima over planes 1..nyu-1
    double m1 = 0.0, m3 = 0.0;
    xrow<NX, XK::value>(
        sm + (size_t)row0 * XK::RS, I.twx, rows, track, m1, m3,
        [&](int pair, int row, const int *k, double2 *A, double2 *B) {
            const int o = row * nxh;
            auto ld = [&](int q, int n1) { return U[q * fs + o + k[n1]]; };
            if (pair == 0) {  // (u1, u3) at the centre
#pragma unroll
                for (int n1 = 0; n1 < KQ; n1++) {
                    A[n1] = ld(0, n1);
                    B[n1] = ld(1, n1);
                }
            } else if (pair == 1) {  // u2 at the centre and at the face
#pragma unroll
                for (int n1 = 0; n1 < KQ; n1++) {
                    A[n1] = ld(-1, n1);
                    B[n1] = ld(2, n1);
                }
#pragma unroll
                for (int n1 = 0; n1 < KQ; n1++)
                    A[n1] = lerp(w0v, B[n1], w1v, A[n1]);
            } else {  // (u1, u3) at the face
                double2 a1[KQ], b1[KQ];
#pragma unroll
                for (int n1 = 0; n1 < KQ; n1++) {
                    A[n1] = ld(3, n1);
                    a1[n1] = ld(0, n1);
                    B[n1] = ld(4, n1);
                    b1[n1] = ld(1, n1);
                }
#pragma unroll
                for (int n1 = 0; n1 < KQ; n1++) {
                    A[n1] = lerp(w0u, A[n1], w1u, a1[n1]);
                    B[n1] = lerp(w0u, B[n1], w1u, b1[n1]);
                }
            }
        },
        [&](int pair, int row, int k, double2 A, double2 B) {
            const int o = 2 * pair * fs + row * nxh + k;
            S[o] = A;
            S[o + fs] = B;
        });
    if (track) xmax(I, m1, m3);
}

// ---------------------------------------------------------------------------
// z forward, masks and derivatives of one (plane, block of cb x modes, half):
// phys_to_four_du's cft (FOU3D.f90:1654-1672), der_x/der_z (:420-523) and
// planes_to_modes_UVP/NUVP.  The six products split into two independent
// halves: {uu, uw, ww} -> Nu1 and Nu3 x/z parts; {vv, uv, wv} -> vv_c, uv_f,
// wv_f and the Nu2 x/z part.  What bounds it: the loads' latency at 22 warps an SM
// and the shared-memory / L1 data pipe (51 % of its cycles at Mz = 192; 56 % while the
// second pass read across banks), whose segments of cb modes are 64 bytes there; wider
// CTAs (up to 512 threads, cb = 10) leave the substep within 2 % or slower.
template <int NZ>
__global__ void __launch_bounds__(LH_ZFWD_T, LH_MINB(NZ, LH_ZFWD_B)) k_zfwd_f(const Inst *__restrict__ insts, const Work *__restrict__ work,
                                                         int count, int cb)
{
    constexpr int N1 = Plan2<NZ>::N1, N2 = Plan2<NZ>::N2;
    constexpr int Nz = 2 * NZ / 3;
    extern __shared__ double2 sm[];
    double2 *T = sm;
    if ((int)blockIdx.x >= count) return;
    const double2 *tw = insts[work[blockIdx.x].inst].twz;  // depends on Mz only
    const int t = threadIdx.x, nv = 3 * cb, v = t % nv, r = t / nv, zb = zblock<NZ>(nv);
    const double2 twr = __ldg(tw + r);  // outer-twiddle base W^r, issued before the data loads
    const int f = v / cb, c = v % cb;
    const FastDiv by_cb(cb);
    {
        const Work w = work[blockIdx.x];
        const Inst &I = insts[w.inst];
        const int nxh = I.nxh, nc = I.nc, j = w.j;
        const int h = w.blk & 1;
        const int i0 = (w.blk >> 1) * cb, i = i0 + c;
        const int g = h == 0 ? (f == 2 ? 3 : f) : (f == 0 ? 2 : f + 3);  // product of this vector
        const double2 *S = sprod_slot(I, w.slot);
        const bool ok = i < nxh;
        if (r < N2) {
            double2 a[N1];
#pragma unroll
            for (int n1 = 0; n1 < N1; n1++)
                a[n1] = ok ? S[((size_t)g * NZ + r + N2 * n1) * nxh + i] : make_double2(0.0, 0.0);
            DFT<N1, -1, NZ>::run(a, tw);
            TwStep ts(twr);
#pragma unroll
            for (int k1 = 0; k1 < N1; k1++) {
                double2 z = a[k1];
                if (k1 > 0) z = twiddle<-1>(ts.next(), z);
                T[k1 * zb + t] = z;
            }
        }
        __syncthreads();
        {
            double2 b[N2];
            if (r < N1) {
#pragma unroll
                for (int n2 = 0; n2 < N2; n2++) b[n2] = T[r * zb + n2 * nv + v];
                DFT<N2, -1, NZ>::run(b, tw);
            }
            __syncthreads();
            if (r < N1) {
                const double dn1 = 1.0 / NZ;
#pragma unroll
                for (int k2 = 0; k2 < N2; k2++) T[(r + N1 * k2) * nv + v] = make_double2(dn1 * b[k2].x, dn1 * b[k2].y);
            }
        }
        __syncthreads();
        for (int e = t; e < Nz * cb; e += blockDim.x) {
            const int kr = by_cb.div(e), cc = by_cb.mod(e, kr), ii = i0 + cc;
            if (ii >= nxh) continue;
            const int zp = kr < Nz / 2 ? kr : kr + NZ - Nz;
            const double2 *row = T + zp * nv + cc;
            const double2 p0 = row[0], p1 = row[cb], p2 = row[2 * cb];
            const size_t on = (size_t)(j - 1) * nc + kr * nxh + ii;
            const bool keep = kr != Nz / 2;  // der_x/der_z zero the kz = -Nz/2 row (FOU3D.f90:444-447)
            const double kx = I.kx[ii], kz = I.kz[kr];
            if (h == 0) {  // p0 uu, p1 uw, p2 ww
                double2 n1 = make_double2(0.0, 0.0), n3 = n1;
                if (keep) {
                    n1 = add_ik(kz, p1, ik(kx, p0));
                    n3 = add_ik(kz, p2, ik(kx, p1));
                }
                I.NXZ1[on] = n1;
                I.NXZ3[on] = n3;
            } else {  // p0 vv, p1 uv, p2 wv
                const size_t o = (size_t)j * nc + kr * nxh + ii;
                I.VVC[o] = p0;
                I.UVF[o] = p1;
                I.WVF[o] = p2;
                double2 n2 = make_double2(0.0, 0.0);
                if (keep) n2 = add_ik(kz, p2, ik(kx, p1));
                I.NXZ2[on] = n2;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// host dispatch
int fast_max_threads(int stage) { return stage == 0 ? LH_ZINV_T : LH_ZFWD_T; }

bool fast_size(int n)
{
    switch (n) {
#define LH_CASE(N) case N:
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
        return true;
    default:
        return false;
    }
}

// Threads one vector of length n uses: max(N1, N2) of its two-pass split.
int fast_vector_threads(int n)
{
    switch (n) {
#define LH_CASE(N) \
    case N:        \
        return Plan2<N>::N1 > Plan2<N>::N2 ? Plan2<N>::N1 : Plan2<N>::N2;
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    default:
        return 0;
    }
}

int fast_threads(int n, int vectors)
{
    int n1 = 1, n2 = 1;
    switch (n) {
#define LH_CASE(N)              \
    case N:                     \
        n1 = Plan2<N>::N1;      \
        n2 = Plan2<N>::N2;      \
        break;
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    default:
        return 0;
    }
    int t = vectors * (n1 > n2 ? n1 : n2);
    return ((t + 31) / 32) * 32;
}

// x stage: z rows per CTA for a bound rb (whole warps, at most kXprodThreads
// lanes), its threads and shared memory
int xprod_rows(int n, int rb)
{
    switch (n) {
#define LH_CASE(N) \
    case N: return XPlan<N>::RW * std::max(1, std::min(kXprodThreads / 32, (rb + XPlan<N>::RW - 1) / XPlan<N>::RW));
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    default: return 1;
    }
}

int xprod_threads(int n, int rb)
{
    switch (n) {
#define LH_CASE(N) \
    case N: return rb / XPlan<N>::RW * 32;
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    default: return 0;
    }
}

size_t xprod_smem(int n, int rb)
{
    switch (n) {
#define LH_CASE(N) \
    case N: return (size_t)rb * XPack<N>::RS * sizeof(double2);
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    default: return 0;
    }
}

// Threads and shared memory of a z-forward CTA of cb x modes (3 cb vectors), shared
// memory of a z-inverse CTA of cb vectors.
int zfwd_threads(int n, int cb) { return fast_threads(n, 3 * cb); }

static size_t exchange_smem(int n, int v)
{
    switch (n) {
#define LH_CASE(N) \
    case N: return (size_t)Plan2<N>::N1 * zblock<N>(v) * sizeof(double2);
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    default: return 0;
    }
}

size_t zfwd_smem(int n, int cb) { return exchange_smem(n, 3 * cb); }

size_t zinv_smem(int n, int cb) { return exchange_smem(n, cb); }

cudaError_t fast_set_attributes(int Mz, int Mx, size_t smz, size_t smx, size_t smf)
{
    cudaError_t e = cudaSuccess;
    switch (Mz) {
#define LH_CASE(N)                                        \
    case N:                                               \
        e = raise_smem_limit((const void *)k_zinv_f<N>, smz); \
        if (e == cudaSuccess) e = raise_smem_limit((const void *)k_zfwd_f<N>, smf); \
        break;
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    default:
        return cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
    switch (Mx) {
#define LH_CASE(N)                                         \
    case N:                                                \
        e = raise_smem_limit((const void *)k_xprod_r<N>, smx); \
        break;
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    default:
        return cudaErrorInvalidValue;
    }
    return e;
}

void fast_launch_zinv(int Mz, unsigned grid, int threads, size_t smem, cudaStream_t st, const Inst *insts,
                      const Work *work, int count, int cb)
{
    switch (Mz) {
#define LH_CASE(N)                                                                   \
    case N:                                                                          \
        k_zinv_f<N><<<grid, threads, smem, st>>>(insts, work, count, cb);       \
        break;
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    }
}

void fast_launch_xprod(int Mx, unsigned grid, int threads, size_t smem, cudaStream_t st, const Inst *insts,
                       const Work *work, int count, int rb, int want_max)
{
    switch (Mx) {
#define LH_CASE(N)                                                                   \
    case N:                                                                          \
        k_xprod_r<N><<<grid, threads, smem, st>>>(insts, work, rb, want_max);        \
        break;
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    }
}

void fast_launch_zfwd(int Mz, unsigned grid, int threads, size_t smem, cudaStream_t st, const Inst *insts,
                      const Work *work, int count, int cb)
{
    switch (Mz) {
#define LH_CASE(N)                                                                   \
    case N:                                                                          \
        k_zfwd_f<N><<<grid, threads, smem, st>>>(insts, work, count, cb);       \
        break;
        LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    }
}

}  // namespace lh
