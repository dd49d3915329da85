// The whole plane pass of a small plane in one CTA: z inverse, x transforms and
// products, z forward with the masks and derivatives, the plane in shared memory
// from the state's rows to the nonlinear terms (modes_to_planes_UVP ..
// planes_to_modes_NUVP, FOU3D.f90:126-261).
//
// The staged kernels (lh_plane_fast.cu) write and read a plane's z-inverse rows
// and products through L2, about seven times the state rows and outputs that a
// plane cannot do without, and take three dependent launches a round; a plane
// of up to 48 x 48 points and its six fields fit half an SM.  Planes share no
// work here, so a plane transforms six rows of fields in z instead of three; the
// operations on each are the staged kernels'.
//
// Layout: P[f][z][i], f = 0 u1(j), 1 u3(j), 2 u2(j-1), 3 u2(j), 4 u1(j+1), 5
// u3(j+1), rows of LDX = nxh | 1 modes.  Every step works in place: a z transform
// exchanges through its own column, the x stage of a row through a matrix of its
// lanes and returns the products uu, uw, vv, ww, uv, wv to the row's six slots (a
// lane reads and writes its own modes only, the face rows first), so only two
// block barriers separate the three steps.
//
// What bounds it: the shared-memory / L1 data pipe, 67 % busy at 16 channels of 32 x
// 32 x 153, and the FP64 pipe, 44 %, at two CTAs an SM (the plane's 78 KB and the row
// matrices).  B200, us a substep, staged -> here:
// 64 channels of 32 x 32 x 153 1515 -> 1239, 16 of them 370 -> 323, 3 of them 92 -> 86, 2
// 58 -> 63; 16 x 16 x 153 alone 33.7 -> 31.5, x 97 28.0 -> 24.5; 32 x 32 x 153 alone,
// whose 152 planes leave four SMs with two, 41.3 -> 46.9 (small_plane_pays decides).
// 288, 320 and 384 threads: 1405, 1435, 1561 us for the 64 where 256 took 1260 (96 and
// 80 registers spill).
#include "lh_fft.cuh"
#include "lh_kernels.cuh"
#include "lh_xprod.cuh"

namespace lh {

constexpr int kSmallThreads = 256;

template <int NX, int NZ>
struct SmallPlane {
    static constexpr int NXH = NX / 3 + 1, LDX = NXH | 1;
    static constexpr int Z1 = NZ == 12 ? 4 : 8, Z2 = NZ / Z1;  // z split; Z1 lanes per vector, Z2 a multiple of 3
    static constexpr int G = kSmallThreads / XPlan<NX>::N1;     // rows of the x stage in flight
    static constexpr size_t plane = (size_t)6 * NZ * LDX;
    static constexpr size_t bytes = (plane + (size_t)G * XPlan<NX>::N1 * XPlan<NX>::LD) * sizeof(double2);
    static_assert(Z2 % 3 == 0 && Z2 <= Z1, "whole k2 rows are kept, every task has its lane");
    static_assert(Z1 == Plan2<NZ>::N1, "the staged kernels' split");
    static_assert(XPlan<NX>::N2 <= XPlan<NX>::N1, "a lane reads and writes the modes of one task");
};

template <int NX, int NZ>
__global__ void __launch_bounds__(kSmallThreads, 2) k_plane_small(const Inst *__restrict__ insts,
                                                                  const Work *__restrict__ work, int want_max)
{
    using SP = SmallPlane<NX, NZ>;
    constexpr int NXH = SP::NXH, LDX = SP::LDX, Z1 = SP::Z1, Z2 = SP::Z2, Nz = 2 * NZ / 3;
    constexpr int FS = NZ * LDX;  // field stride in P
    extern __shared__ double2 sm[];
    double2 *const P = sm;
    const Work w = work[blockIdx.x];
    const Inst &I = insts[w.inst];
    const int t = threadIdx.x, j = w.j, nc = I.nc;
    const double2 *const twz = I.twz;
    const int rz = t % Z1, gz = t / Z1;  // lane and group of the z steps
    constexpr int GZ = kSmallThreads / Z1;
    const int wz = (t & ~31) / Z1;  // first group of this warp

    // ---- z inverse: vectors (field, x mode), the pruned cft of four_to_phys_u ----
    {
        const size_t row = (size_t)j * nc;
        const double2 base = __ldg(twz + rz);
#pragma unroll 1
        for (int v0 = 0; v0 < 6 * NXH; v0 += GZ) {
            if (v0 + wz >= 6 * NXH) break;  // nothing left for this warp
            const int v = v0 + gz, f = v / NXH, i = v % NXH;
            const bool act = v < 6 * NXH;
            double2 *const T = P + f * FS + i;
            const double2 *X = (f == 0 || f == 4 ? I.U1 : (f == 1 || f == 5 ? I.U3 : I.U2)) + row;
            if (f == 2) X -= nc;
            if (f >= 4) X += nc;
            if (act && rz < Z2) {
                double2 a[Z1];
#pragma unroll
                for (int n1 = 0; n1 < Z1; n1++) {
                    const int n = rz + Z2 * n1, kr = n < Nz / 2 ? n : n - NZ / 3;
                    a[n1] = n < Nz / 2 || n >= NZ - Nz / 2 ? X[kr * NXH + i] : make_double2(0.0, 0.0);
                }
                DFT<Z1, +1, NZ>::run(a, twz);
                TwStep ts(base);
#pragma unroll
                for (int k1 = 0; k1 < Z1; k1++)
                    T[(k1 * Z2 + rz) * LDX] = k1 > 0 ? twiddle<+1>(ts.next(), a[k1]) : a[k1];
            }
            __syncwarp();
            double2 b[Z2];
            if (act) {
#pragma unroll
                for (int n2 = 0; n2 < Z2; n2++) b[n2] = T[(rz * Z2 + n2) * LDX];
                DFT<Z2, +1, NZ>::run(b, twz);
            }
            __syncwarp();
            if (act) {
#pragma unroll
                for (int k2 = 0; k2 < Z2; k2++) T[(rz + Z1 * k2) * LDX] = b[k2];
            }
        }
    }
    __syncthreads();

    // ---- x transforms and products, row by row ----------------------------------
    {
        using XP = XPlan<NX>;
        const int g = t / XP::N1;
        double2 *const T = sm + SP::plane + (size_t)g * XP::N1 * XP::LD;
        const bool track = want_max && I.dt_mode == 0 && j <= I.nyu - 1;
        const double dnv = 1.0 / (I.yv[j] - I.yv[j - 1]), dnu = 1.0 / (I.yu[j + 1] - I.yu[j]);
        const double w0v = (I.yu[j] - I.yv[j - 1]) * dnv, w1v = (I.yv[j] - I.yu[j]) * dnv;
        const double w0u = (I.yv[j] - I.yu[j]) * dnu, w1u = (I.yu[j + 1] - I.yv[j]) * dnu;
        double m1 = 0.0, m3 = 0.0;
#pragma unroll 1
        for (int z0 = 0; z0 < NZ; z0 += SP::G) {
            if (z0 + (t & ~31) / XP::N1 >= NZ) break;  // nothing left for this warp
            const int z = z0 + g;
            const bool rowok = z < NZ;
            double2 *const row = P + (rowok ? z : 0) * LDX;
            double2 FA[XP::KQ], FB[XP::KQ];  // (u1, u3) at the face, interpolated before pair 0's products take its slots
            xrow<NX, false>(
                T, I.twx, rowok, track, m1, m3,
                [&](int pair, int, const int *k, double2 *A, double2 *B) {
                    if (pair == 0) {
#pragma unroll
                        for (int n1 = 0; n1 < XP::KQ; n1++) {
                            A[n1] = row[k[n1]];
                            B[n1] = row[FS + k[n1]];
                            const double2 a0 = row[4 * FS + k[n1]], b0 = row[5 * FS + k[n1]];
                            FA[n1] = lerp(w0u, a0, w1u, A[n1]);
                            FB[n1] = lerp(w0u, b0, w1u, B[n1]);
                        }
                    } else if (pair == 1) {
#pragma unroll
                        for (int n1 = 0; n1 < XP::KQ; n1++) {
                            A[n1] = row[2 * FS + k[n1]];
                            B[n1] = row[3 * FS + k[n1]];
                            A[n1] = lerp(w0v, B[n1], w1v, A[n1]);
                        }
                    } else {
#pragma unroll
                        for (int n1 = 0; n1 < XP::KQ; n1++) A[n1] = FA[n1], B[n1] = FB[n1];
                    }
                },
                [&](int pair, int, int k, double2 A, double2 B) {
                    row[2 * pair * FS + k] = A;
                    row[(2 * pair + 1) * FS + k] = B;
                });
        }
        if (track) xmax(I, m1, m3);
    }
    __syncthreads();

    // ---- z forward, masks and derivatives: (half, x mode) per Z1 lanes ------------
    const double2 base = __ldg(twz + rz);
#pragma unroll 1
    for (int v0 = 0; v0 < 2 * NXH; v0 += GZ) {
        if (v0 + wz >= 2 * NXH) break;  // nothing left for this warp
        const int v = v0 + gz, h = v / NXH, i = v % NXH;
        const bool act = v < 2 * NXH;
        // products of this half, in order: uu, uw, ww or vv, uv, wv
        double2 *const T0 = P + (h ? 2 : 0) * FS + i, *const T1 = P + (h ? 4 : 1) * FS + i, *const T2 = P + (h ? 5 : 3) * FS + i;
        if (act && rz < Z2) {
#pragma unroll 1
            for (int p = 0; p < 3; p++) {
                double2 *const T = p == 0 ? T0 : (p == 1 ? T1 : T2);
                double2 a[Z1];
#pragma unroll
                for (int n1 = 0; n1 < Z1; n1++) a[n1] = T[(rz + Z2 * n1) * LDX];
                DFT<Z1, -1, NZ>::run(a, twz);
                TwStep ts(base);
                // element n1 of this lane's set is only its own until the exchange
#pragma unroll
                for (int k1 = 0; k1 < Z1; k1++)
                    T[(rz + Z2 * k1) * LDX] = k1 > 0 ? twiddle<-1>(ts.next(), a[k1]) : a[k1];
            }
        }
        __syncwarp();
        if (act) {
            const double dn1 = 1.0 / NZ, kx = I.kx[i];
            // kept rows: k = rz + Z1 k2 for k2 < Z2/3 (row k) and k2 >= 2 Z2/3 (row k -
            // NZ/3); der_x/der_z zero the kz = -Nz/2 row (FOU3D.f90:444-447), k = 2 NZ/3
            constexpr int KE = 2 * Z2 / 3;
            double2 b[Z2], acc[KE];
            auto pass = [&](const double2 *T) {
#pragma unroll
                for (int n2 = 0; n2 < Z2; n2++) b[n2] = T[(n2 + Z2 * rz) * LDX];
                DFT<Z2, -1, NZ>::run(b, twz);
#pragma unroll
                for (int e = 0; e < KE; e++) {
                    const double2 p = b[e < Z2 / 3 ? e : e + Z2 / 3];
                    b[e] = make_double2(dn1 * p.x, dn1 * p.y);
                }
            };
            auto add_dx = [&]() {
#pragma unroll
                for (int e = 0; e < KE; e++) acc[e] = ik(kx, b[e]);
            };
            const size_t o = (size_t)j * nc + rz * NXH + i;  // row e of this lane: Z1 e rows further
            auto add_dz_store = [&](double2 *X) {
#pragma unroll
                for (int e = 0; e < KE; e++) {
                    const double kz = I.kz[rz + Z1 * e];
                    double2 n = add_ik(kz, b[e], acc[e]);
                    if (rz == 0 && e == Z2 / 3) n = make_double2(0.0, 0.0);
                    X[o - nc + Z1 * e * NXH] = n;
                }
            };
            auto store = [&](double2 *X) {
#pragma unroll
                for (int e = 0; e < KE; e++) X[o + Z1 * e * NXH] = b[e];
            };
            pass(T0);
            if (h) store(I.VVC);
            else add_dx();
            pass(T1);
            if (h) store(I.UVF);
            else add_dz_store(I.NXZ1);
            add_dx();
            pass(T2);
            if (h) store(I.WVF);
            add_dz_store(h ? I.NXZ2 : I.NXZ3);
        }
    }
}

#define LH_SMALL_PLANES(X) X(12, 12) X(12, 24) X(12, 48) X(24, 12) X(24, 24) X(24, 48) X(48, 12) X(48, 24) X(48, 48)

bool small_plane(int Mx, int Mz)
{
#define LH_CASE(A, B) \
    if (Mx == A && Mz == B) return true;
    LH_SMALL_PLANES(LH_CASE)
#undef LH_CASE
    return false;
}

// Whether the one-CTA pass is the faster one for `planes` planes in a plan.  The
// same bits either way.  Planes of up to 24 x 48 points: always; 48 x 48: 256
// planes 58.4 us a substep against 59.4 staged, 304 63.3 against 58.3, 456 85.8
// against 91.4, 1216 207 against 228.
bool small_plane_pays(int Mx, int Mz, long planes)
{
    return small_plane(Mx, Mz) && (Mx * Mz <= 24 * 48 || planes >= 400);
}

cudaError_t small_plane_attributes(int Mx, int Mz)
{
#define LH_CASE(A, B) \
    if (Mx == A && Mz == B) return raise_smem_limit((const void *)k_plane_small<A, B>, SmallPlane<A, B>::bytes);
    LH_SMALL_PLANES(LH_CASE)
#undef LH_CASE
    return cudaErrorInvalidValue;
}

void small_plane_launch(int Mx, int Mz, unsigned grid, cudaStream_t st, const Inst *insts, const Work *work, int want_max)
{
#define LH_CASE(A, B)      \
    if (Mx == A && Mz == B) \
        k_plane_small<A, B><<<grid, kSmallThreads, SmallPlane<A, B>::bytes, st>>>(insts, work, want_max);
    LH_SMALL_PLANES(LH_CASE)
#undef LH_CASE
}

}  // namespace lh
