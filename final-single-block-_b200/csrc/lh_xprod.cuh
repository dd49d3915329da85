// The x stage of a z row, shared by the staged plane kernels (lh_plane_fast.cu)
// and the one-CTA plane pass (lh_plane_small.cu).
#pragma once

#include "lh_fft.cuh"

namespace lh {

// Operations that the staged and the one-CTA plane kernels share, with their
// roundings spelled out, so that a plane is the same bits by either.
// w0 x + w1 y: the y interpolations
__device__ __forceinline__ double2 lerp(double w0, double2 x, double w1, double2 y)
{
    return make_double2(fma(w0, x.x, w1 * y.x), fma(w0, x.y, w1 * y.y));
}
// i k p, and a + i k p: der_x, der_z
__device__ __forceinline__ double2 ik(double k, double2 p) { return make_double2(-(k * p.y), k * p.x); }
__device__ __forceinline__ double2 add_ik(double k, double2 p, double2 a)
{
    return make_double2(fma(-k, p.y, a.x), fma(k, p.x, a.y));
}

// Outer twiddles W^(r k1), k1 = 1.., of a two-pass transform by the
// recurrence W^(r k1) = W^(r (k1-1)) W^r from one table entry, which keeps the
// per-point table reads out of the shared-memory pipe (the kernels' busiest
// unit); the recurrence's rounding stays within a few ulp for k1 <= 24.
struct TwStep {
    double2 w1, wk;
    __device__ explicit TwStep(double2 base) : w1(base), wk(make_double2(1.0, 0.0)) {}
    __device__ __forceinline__ double2 next()
    {
        wk = make_double2(fma(wk.x, w1.x, -(wk.y * w1.y)), fma(wk.x, w1.y, wk.y * w1.x));
        return wk;
    }
};

// ---------------------------------------------------------------------------
// x transforms and products of one z row of a plane, the products in registers.  N1 lanes of a warp own a z row and take its three vectors (pairs)
// in turn; NX = N1 N2.
//
//   gather   the lane of task n2 loads the modes k = n2 + N2 q <= Nx/2 of the
//            pair's two real rows A, B (with the y interpolations), forms z[k] =
//            A + iB for itself and z[NX - k] = conj(A) + i conj(B) for the lane
//            of task N2 - n2 (one shuffle), so the inputs of the inverse
//            transform never pass through shared memory;
//   inverse  DFT over N1, twiddle, exchange through the row's N1 x N2 matrix,
//            DFT over N2: lane r holds the physical values x = r + N1 t;
//   products in registers: u3^2 of the first pair waits for the second, u2 of
//            the second for the third;
//   forward  the mirrored split (DFT over N2 first, in the registers that hold
//            the products), exchange, DFT over N1: the lane of task m holds the
//            modes k = m + N2 q;
//   split    the packed real transforms need Z[NX - k], on the lane of task
//            N2 - m: one shuffle again; modes i <= Nx/2 are stored.
//
// A vector crosses shared memory twice (the exchanges, 4 accesses an element)
// instead of 12 accesses when the gather, the products and the split went
// through it too.  That pipe was still the busiest (57 % of its cycles at Mx = 192,
// against the FP64 pipe's 50 %), so the tasks of as many whole rows as fit sit on
// consecutive lanes (24 of 32 at N2 = 12; on the rows' own lanes they took four
// wavefronts an access instead of three), m -> N2 - m stays inside the row, and the
// matrices of neighbouring rows are a task's columns apart in the banks (now 50 % and
// 51 %, wavefronts of a substep at 128^2 x 153 21.5 -> 18.3 million).  A lane
// keeps its columns of the matrix from one use to the next, so two __syncwarp a
// vector are all the synchronisation.  Every load of a task is issued before the
// first is used: loaded mode by mode the stage waited on L2 for half its time.
template <int NX>
struct XPlan {
    // the substep at the other splits, us: 192 as 8 x 24 394 (16 x 12: 362), 144 as
    // 8 x 18 153 (148), 96 as 4 x 24 129 and 16 x 6 123 (114), 48 as 4 x 12 51 (44)
    static constexpr int N1 = NX == 12                                         ? 4
                              : (NX == 36 || NX == 54 || NX == 162)            ? 6
                              : (NX == 24 || NX == 48 || NX == 72 || NX == 96) ? 8
                              : (NX == 108 || NX == 216 || NX == 324)          ? 12
                                                                               : 16;
    static constexpr int N2 = NX / N1;
    static constexpr int LD = N2 | 1;             // odd row stride: conflict-free rows and columns
    static constexpr int KQ = NX / 3 / N2 + 1;    // modes k <= Nx/2 of a task, at most
    static constexpr int RW = 32 / N1;            // rows per warp; N1 = 6 and 12 leave lanes over
    static constexpr bool WHOLE = RW * N1 == 32;
    static_assert(N1 * N2 == NX && N1 % 2 == 0 && 2 * KQ <= N1 + 1, "modes, mirror images, zeros between");
};
// Whether the tasks of RPR whole rows are packed on a warp's consecutive lanes or
// every row's stay on its own N1 lanes: packed where they do not fit those, or touch
// fewer groups of eight lanes (a quarter of an access's wavefronts each) that way.
template <int NX>
struct XPack {
    using XP = XPlan<NX>;
    static constexpr int N1 = XP::N1, N2 = XP::N2, RW = XP::RW;
    static constexpr int groups()
    {
        int n = 0;
        for (int g = 0; g < 4; g++)
            for (int l = 8 * g; l < 8 * g + 8; l++)
                if (l < RW * N1 && l % N1 < N2) {
                    n++;
                    break;
                }
        return n;
    }
    static constexpr bool value = N2 > N1 || (RW * N2 + 7) / 8 < groups();
    static constexpr int RPR = 32 / N2 < RW ? 32 / N2 : RW;
    // elements from one row's matrix to the next: in the banks the tasks of
    // neighbouring rows follow one another (the lanes of the middle pass do where
    // those cannot)
    static constexpr int RS = N1 * XP::LD + (value ? ((RPR > 1 && (N1 % 8 == 0 || N1 >= N2) ? N2 : N1 * XP::LD) - N1 * XP::LD) & 7 : 0);
};

// The three pairs of a warp's RW rows: load(pair, row, k, A, B) fetches the modes k[]
// of the two real rows, store(pair, row, k, A, B) takes the spectra of the two
// products at mode k.  PACKED: T the warp's exchange matrices, RS apart, rows how many
// of the rows there are.  Otherwise T is the matrix of this lane's row, rows whether
// it exists, and row always 0.  m1, m3 gather max |u1|, |u3| when track.  Every lane
// of the warp calls it.
template <int NX, bool PACKED, class Load, class Store>
__device__ __forceinline__ void xrow(double2 *T, const double2 *tw, int rows, bool track, double &m1, double &m3,
                                     Load &&load, Store &&store)
{
    using XP = XPlan<NX>;
    constexpr int N1 = XP::N1, N2 = XP::N2, LD = XP::LD, KQ = XP::KQ, nxh = NX / 3 + 1;
    constexpr int RW = XP::RW, RPR = PACKED ? XPack<NX>::RPR : RW, RS = XPack<NX>::RS, ROUNDS = (RW + RPR - 1) / RPR;
    static_assert(PACKED || N2 <= N1, "a lane for every task");
    const int lane = threadIdx.x & 31, r = lane % N1, lane_row = lane / N2, lane_task = lane - lane_row * N2;
    const bool on = XP::WHOLE || lane < RW * N1;
    double2 *const Tr = T + ((PACKED && on ? lane / N1 * RS : 0) + r * LD);  // row r of the matrix, the middle pass
    // task m of `row`, the lane of task N2 - m.  What follows from packed ones is formed
    // again in each round: kept for all three pairs it would spill.
    struct Task {
        int m, partner, row;
        bool on, ok;
        __device__ Task(int g, int tl, int tm, int r, bool lane_on, int rows) : m(tm), row(0)
        {
            if (PACKED) {
                asm volatile("" : "+r"(tl), "+r"(m));
                partner = tl * N2 + (m > 0 ? N2 - m : 0);
                row = g * RPR + tl;
                on = tl < RPR && (RW % RPR == 0 || row < RW);
                ok = on && row < rows;
            } else {
                m = r < N2 ? r : -1;
                partner = (int)(threadIdx.x & 31) - r + (r < N2 ? (N2 - r) % N2 : r);
                on = m >= 0 && lane_on;
                ok = on && rows != 0;
            }
        }
    };
    double saved[N2];
#pragma unroll 1
    for (int pair = 0; pair < 3; pair++) {
        // gather and inverse pass 1
#pragma unroll 1
        for (int g = 0; g < ROUNDS; g++) {
            const Task q(g, lane_row, lane_task, r, on, rows);
            double2 *const Tm = T + (q.row * RS + q.m);
            double2 a[N1], mir[KQ], A[KQ], B[KQ];
            // every load of the task before the first use (indices past the
            // modes are clamped, their values dropped)
            int kk[KQ];
#pragma unroll
            for (int n1 = 0; n1 < KQ; n1++) {
                const int k = (q.m >= 0 ? q.m : 0) + N2 * n1;
                kk[n1] = k < nxh ? k : 0;
            }
            load(pair, q.ok ? q.row : 0, kk, A, B);
#pragma unroll
            for (int k1 = 0; k1 < N1; k1++) a[k1] = make_double2(0.0, 0.0);
#pragma unroll
            for (int n1 = 0; n1 < KQ; n1++) {
                const int k = q.m + N2 * n1;
                const bool in = q.ok && k < nxh;
                if (!in) A[n1] = B[n1] = make_double2(0.0, 0.0);
                if (k == 0) A[n1].y = B[n1].y = 0.0;  // Im of mode 0 dropped (rft_buff.f:78-81)
                a[n1] = make_double2(A[n1].x - B[n1].y, A[n1].y + B[n1].x);
                mir[n1] = make_double2(A[n1].x + B[n1].y, B[n1].x - A[n1].y);
            }
#pragma unroll
            for (int n1 = 0; n1 < KQ; n1++) {
                const double2 z = make_double2(__shfl_sync(0xffffffffu, mir[n1].x, q.partner),
                                               __shfl_sync(0xffffffffu, mir[n1].y, q.partner));
                // z[NX - k] sits at N1 - 1 - n1 on the partner; task 0 is its own, one higher
                const double2 own = n1 + 1 < KQ ? mir[n1 + 1] : make_double2(0.0, 0.0);
                a[N1 - 1 - n1] = q.m == 0 ? own : z;
            }
            DFT<N1, +1, NX>::run(a, tw);
            if (q.on) {
                TwStep ts(__ldg(tw + q.m));
#pragma unroll
                for (int k1 = 0; k1 < N1; k1++) Tm[k1 * LD] = k1 > 0 ? twiddle<+1>(ts.next(), a[k1]) : a[k1];
            }
        }
        __syncwarp();
        // inverse pass 2, products, forward pass 1 of this lane's row of the matrix.  Lanes
        // left over (N1 = 6, 12) take no part: rows are overwritten here without a barrier,
        // so nobody but their lanes may read them.
        if (on) {
            double2 b[N2];
#pragma unroll
            for (int n2 = 0; n2 < N2; n2++) b[n2] = Tr[n2];
            DFT<N2, +1, NX>::run(b, tw);
            if (pair == 0) {
#pragma unroll
                for (int x = 0; x < N2; x++) {
                    const double u1 = b[x].x, u3 = b[x].y;
                    if (track) {
                        m1 = fmax(m1, fabs(u1));
                        m3 = fmax(m3, fabs(u3));
                    }
                    saved[x] = u3 * u3;
                    b[x] = make_double2(u1 * u1, u1 * u3);
                }
            } else if (pair == 1) {
#pragma unroll
                for (int x = 0; x < N2; x++) {
                    const double u2c = b[x].x, u2 = b[x].y;
                    b[x] = make_double2(u2c * u2c, saved[x]);
                    saved[x] = u2;
                }
            } else {
#pragma unroll
                for (int x = 0; x < N2; x++) b[x] = make_double2(b[x].x * saved[x], b[x].y * saved[x]);
            }
            DFT<N2, -1, NX>::run(b, tw);
            TwStep ts(__ldg(tw + r));
#pragma unroll
            for (int n2 = 0; n2 < N2; n2++) Tr[n2] = n2 > 0 ? twiddle<-1>(ts.next(), b[n2]) : b[n2];
        }
        __syncwarp();
        // forward pass 2, split, scale 1/Mx
#pragma unroll 1
        for (int g = 0; g < ROUNDS; g++) {
            const Task q(g, lane_row, lane_task, r, on, rows);
            const int m = q.m;
            // packed lanes without a task read nothing, others a column whose values they drop
            const double2 *const Tm = T + (q.row * RS + (m >= 0 ? m : 0));
            double2 e[N1];
#pragma unroll
            for (int k1 = 0; k1 < N1; k1++) e[k1] = !PACKED || q.on ? Tm[k1 * LD] : make_double2(0.0, 0.0);
            DFT<N1, -1, NX>::run(e, tw);
            const double h = 0.5 / NX;
#pragma unroll
            for (int k1 = 0; k1 < KQ; k1++) {
                const double2 z = make_double2(__shfl_sync(0xffffffffu, e[N1 - 1 - k1].x, q.partner),
                                               __shfl_sync(0xffffffffu, e[N1 - 1 - k1].y, q.partner));
                const int k = m + N2 * k1;
                const double2 zk = e[k1], own = e[(N1 - k1) % N1], zm = m == 0 ? own : z;
                if (q.ok && k < nxh) {
                    double2 A = make_double2(h * (zk.x + zm.x), h * (zk.y - zm.y));
                    double2 B = make_double2(h * (zk.y + zm.y), h * (zm.x - zk.x));
                    if (k == 0) A.y = B.y = 0.0;
                    store(pair, q.row, k, A, B);
                }
            }
        }
    }
}

// CFL maxima of a warp's rows into the instance (rows past the last are zero).
__device__ __forceinline__ void xmax(const Inst &I, double m1, double m3)
{
    for (int o = 16; o > 0; o >>= 1) {
        m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
        m3 = fmax(m3, __shfl_xor_sync(0xffffffffu, m3, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(reinterpret_cast<unsigned long long *>(&I.sc[SC_U1MAX]), (unsigned long long)__double_as_longlong(m1));
        atomicMax(reinterpret_cast<unsigned long long *>(&I.sc[SC_U3MAX]), (unsigned long long)__double_as_longlong(m3));
    }
}

}  // namespace lh
