// Column pass of one RK3 substep for plans of few columns: tiles of C columns
// held in shared memory from the right-hand sides to the corrected state, the y
// rows spread over the lanes.
//
// The operations are those of k_column (lh_column.cu), whose recurrences take
// one step per row on one lane per column: with few columns most SMs idle and
// four sweeps of 150 and more steps set the pace.  Here a CTA keeps the three
// velocity systems of its C columns on chip and every recurrence is cut into
// L = 32 blocks of rows: a lane composes the affine maps of its block, a
// scan over the blocks gives the value entering each, and the lane runs its
// rows with the reference's per-row arithmetic.  Only the values at block
// boundaries are formed in another order (a few ulp).  The LU factors depend on
// dt alone, so k_factors forms them beside the plane pass.
//
// What bounds it: the dependent chain of one CTA (about 43,000 cycles at 153 rows and 8
// columns, a third of its waits on the right-hand sides' loads), and a large code run once;
// so a lane works on the three systems at once, three independent chains, its
// next row's loads in flight, and the loops stay rolled (unrolled to 108 KB of
// code the pass was half again as slow).  Column pass alone, us a substep on
// B200, k_column -> tiles: 32x32x153 86 -> 23, 64x64x153 94 -> 51, 96x64x129
// 85 -> 65; the whole substep, with the per-column kernel that served up to 1536
// columns before the tiles in brackets: 16x16x97 61 [30] -> 24, 32x32x153 99
// [52] -> 41, 32x32x257 156 [104] -> 59, 64x64x153 149 -> 111.  Larger plans keep
// k_column, whose streaming sweeps move half again as many rows once they fill
// the GPU (tile_columns, lh_engine.cu).
//
// Phases (lane = column + C * row block; a lane owns the same rows in every phase,
// so shared memory between the phases is its own but for one u2 row):
//   1  the pivots and the DG factors land in shared memory by cp.async, the first
//      rows in registers
//   2  right-hand sides (RHS0, Nu sum, du += -g Nu, solveU rhs) of u1, u3 and
//      u2, with the forward eliminations composed on the way; eliminations with
//      the back substitutions composed on the way; back substitutions
//   3  divergence and the LUsolP forward sweep, then its back sweep with p +=
//      psi, v_corr and the ghost rows, so psi is never stored and every row of
//      the state is written once
#include "lh_column.cuh"

namespace lh {

constexpr int kTileBlocks = 32;  // row blocks, the lanes that share a column

// y -> A + B y with complex A, real B: a block of a forward or back
// substitution.  N systems side by side; the first two share B when N = 3 (u1
// and u3 have the same matrix).
template <int N>
struct Aff {
    static constexpr int kB = N == 3 ? 2 : 1;
    double2 A[N];
    double B[kB];
    __device__ static constexpr int b(int k) { return k == 2 ? 1 : 0; }
    __device__ __forceinline__ void reset()
    {
#pragma unroll
        for (int k = 0; k < N; k++) A[k] = make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < kB; k++) B[k] = 1.0;
    }
    // this map after x
    __device__ __forceinline__ double2 at(int k, double2 x) const
    {
        return make_double2(fma(B[b(k)], x.x, A[k].x), fma(B[b(k)], x.y, A[k].y));
    }
};

// Values entering each row block of affine chains: the composition of the maps
// of all blocks before this one (up, ascending rows) or after it, over the
// kTileBlocks blocks of a column: a scan inside segments of four blocks (lanes
// of one warp, whatever C is, so the order of the operations does not depend on
// it), then the totals of the segments before, which pass through `part`
// ([kTileBlocks / 4][C], a different one in consecutive scans: the barrier of
// the scan between them separates its readers from its next writers).  On
// return m.A holds the entering values.
template <int C, int N>
__device__ __noinline__ Aff<N> scan_entry(Aff<N> m, Aff<N> *part, bool up)
{
    constexpr int NS = kTileBlocks / 4;
    const int lane = threadIdx.x & 31, c = threadIdx.x % C, b = threadIdx.x / C;
    const int pos = up ? b % 4 : 3 - b % 4, seg = up ? b / 4 : NS - 1 - b / 4;  // in sweep order
#pragma unroll 1
    for (int o = 1; o <= 4; o <<= 1) {
        // the last round makes the scan exclusive
        if (o == 4 && pos == 3) part[seg * C + c] = m;
        const int dist = o == 4 ? C : o * C, src = (up ? lane - dist : lane + dist) & 31;
        Aff<N> f;
#pragma unroll
        for (int k = 0; k < N; k++)
            f.A[k] = make_double2(__shfl_sync(0xffffffffu, m.A[k].x, src), __shfl_sync(0xffffffffu, m.A[k].y, src));
#pragma unroll
        for (int k = 0; k < Aff<N>::kB; k++) f.B[k] = __shfl_sync(0xffffffffu, m.B[k], src);
        if (o == 4) {
            m = f;
            if (pos == 0) m.reset();
        } else if (pos >= o) {
#pragma unroll
            for (int k = 0; k < N; k++) m.A[k] = m.at(k, f.A[k]);
#pragma unroll
            for (int k = 0; k < Aff<N>::kB; k++) m.B[k] *= f.B[k];
        }
    }
    __syncthreads();
    double2 v[N];
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < NS - 1; q++) {
        if (q < seg) {
            const Aff<N> &f = part[q * C + c];
#pragma unroll
            for (int k = 0; k < N; k++) v[k] = f.at(k, v[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < N; k++) m.A[k] = m.at(k, v[k]);
    return m;
}

// Bit-exact block entries.  The flow-rate correction divides a difference of
// two flow rates by dt, so the last bits of the mean mode count: in the tile
// that holds it the entries of u1 are refined until they reproduce themselves.
// sweep(x) runs a block from entry x and returns its exit; the exit of the
// neighbouring block (its own rows before in sweep order) is the next entry.
// When no entry changes any more the sweeps equal the sequential ones bit for
// bit; the recurrences contract, so one or two rounds do, and L rounds always do.
__device__ __forceinline__ bool same_bits(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
template <int C, bool UP, class Sweep>
__device__ __forceinline__ double2 exact_entries(double2 x, double2 *part, Sweep &&sweep)
{
    constexpr int L = kTileBlocks;
    const int t = threadIdx.x, b = t / C;
    __syncthreads();  // a scan may still be reading part
#pragma unroll 1
    for (int it = 0; it < L; it++) {
        part[t] = sweep(x);
        __syncthreads();
        const double2 y = b == (UP ? 0 : L - 1) ? x : part[UP ? t - C : t + C];
        const bool moved = !(same_bits(x.x, y.x) && same_bits(x.y, y.y));
        x = y;
        if (!__syncthreads_or(moved)) break;
    }
    return x;
}

// Shared memory of a tile: three systems, the pivots (psi later takes their
// place), DG2 and DG3, scan totals (two sets), y metrics.
constexpr int tile_scan_doubles(int C) { return 2 * (kTileBlocks / 4) * C * 8; }
static_assert(tile_scan_doubles(1) >= 2 * kTileBlocks, "the block exits of exact_entries fit the totals' space");
size_t column_tile_smem_bytes(int nyu, int C)
{
    const size_t R = (size_t)nyu + 1;
    return (4 * R * C * 2 + 2 * nyu * C + tile_scan_doubles(C) + 9 * (R + 1)) * sizeof(double);
}

// Columns per tile of an instance of nyu rows in a plan of total columns; 0:
// the tiles do not serve it.  An SM holds 8 columns at a time (the registers of
// 32 lanes each) however they are cut into tiles, so narrow tiles spread few
// columns over more SMs, and wide ones read whole lines: 2 up to two columns an
// SM, 4 up to 1184 columns, one wave, then 8, narrower where the rows do not
// fit shared memory.  The width does not change the arithmetic.
int column_tile_width(int nyu, int nc, size_t total)
{
    if ((size_t)nc * (nyu + 2) > (1u << 27)) return 0;  // 32-bit offsets over the instance's fields
    for (int C = total <= 2 * 148 ? 2 : (total <= 8 * 148 ? 4 : 8); C >= 2; C /= 2)
        if (column_tile_smem_bytes(nyu, C) <= 220 * 1024) return C;
    return 0;
}

// x -> (a x + b) / (c x + d), the LU-factor step a3u' = a3 / (a2 - a1 a3u)
struct Mob {
    double a, b, c, d;
};
// Scale a map by a power of two (exact; the map is homogeneous) so that long
// products stay in range.
__device__ __forceinline__ void mob_rescale(Mob &m)
{
    const int hi = __double2hiint(fmax(fmax(fabs(m.a), fabs(m.b)), fmax(fabs(m.c), fabs(m.d))));
    const int e = hi >> 20;  // biased exponent of the largest entry
    if (e <= 0 || e >= 0x7fe) return;
    const double s = __hiloint2double((0x7fe - e) << 20, 0);
    m.a *= s;
    m.b *= s;
    m.c *= s;
    m.d *= s;
}

// The power of two that brings the interior rows of a stiff column to about one: at time
// steps where a row's entries pass 1e30 the product of eight or nine maps would leave
// the range of a double, though the recurrence does not.  1 otherwise.
__device__ __forceinline__ double helm_scale(double beta, const double *d, double k2x, double k2z)
{
    const int e = __double2hiint(fabs(beta) * (fabs(d[4]) + fabs(k2x) + fabs(k2z))) >> 20;
    return e < 0x3ff + 100 || e >= 0x7fe ? 1.0 : __hiloint2double((0x7fe - e) << 20, 0);
}

// Inverse pivots of the Helmholtz systems of one grid (w.blk: 0 u, 1 v) for
// kFactorColumns columns: LU_build + LU_dec (tridLU_3D.f90:163-221, 327-364).
// Bound by the length of the chain, one division a row, so kFactorBlocks lanes
// share a column: each composes the 2x2 maps of its block of rows, the products
// of the blocks below give the scaled upper diagonal entering it, and its rows
// run by the reference's recurrence.  For the mean mode of a constant-flow-rate
// run (exact_entries) the entries are then refined until they reproduce
// themselves, so that its pivots are the sequential ones bit for bit.  One lane
// a column took 24 us at 154 rows, longer than the plane pass of a small
// channel that it runs beside.
__global__ void __launch_bounds__(kFactorColumns *kFactorBlocks) k_factors(const Inst *__restrict__ insts,
                                                                           const Work *__restrict__ work, int kRK)
{
    constexpr int C = kFactorColumns, L = kFactorBlocks, T = C * L;
    extern __shared__ double sd[];  // the grid's d2/dy2 coefficients
    __shared__ Mob maps[T];
    __shared__ double ends[T];
    const Work w = work[blockIdx.x];
    const Inst &I = insts[w.inst];
    const bool v = w.blk != 0;
    const int n = v ? I.nyv : I.nyu, nc = I.nc, nxh = I.nxh;
    const double *d = v ? I.dyv2i : I.dyu2i;
    for (int e = threadIdx.x; e < 3 * (n + 1); e += T) sd[e] = d[e];
    const int t = threadIdx.x, b = t / C, col = min(w.j * C + t % C, nc - 1);
    const double k2x = I.k2x[col % nxh], k2z = I.k2z[col / nxh];
    // the fixed dt is also what SC_DT holds; k_dt may be writing it meanwhile
    const double beta = rk_coeffs(kRK).b * (I.dt_mode == 0 ? I.sc[SC_DT] : I.dt_fixed) / I.Re;
    const double w0 = v ? 0.0 : I.gw1, wt = v ? 0.0 : I.gw2;
    const int K = (n + L - 1) / L, r0 = min(n + 1, 1 + b * K), r1 = min(n + 1, r0 + K);  // interior rows of the block
    __syncthreads();
    Mob m{1.0, 0.0, 0.0, 1.0};
    // stiff columns row by row: times the scale, the rows took 8 more registers (five CTAs an SM)
    const int every = helm_scale(beta, sd, k2x, k2z) != 1.0 ? 0 : 7;
#pragma unroll 1
    for (int j = r0; j < r1; j++) {
        const HRow h = helm_row(j, n, sd, beta, k2x, k2z, w0, wt);
        m = Mob{h.a3 * m.c, h.a3 * m.d, fma(h.a2, m.c, -h.a1 * m.a), fma(h.a2, m.d, -h.a1 * m.b)};
        if (((j - r0) & every) == every) mob_rescale(m);
    }
    mob_rescale(m);
    maps[t] = m;
    __syncthreads();
    double p = w0 * 1.0, q = 1.0;  // the entering value as p / q, from row 0
#pragma unroll 4
    for (int k = t % C; k < t; k += C) {
        const Mob f = maps[k];
        const double r = fma(f.a, p, f.b * q);
        q = fma(f.c, p, f.d * q);
        p = r;
    }
    double x = p / q;
    auto pivot = [&](int j, double &x) {
        const double a1 = -beta * sd[3 * j], a2 = 1.0 - beta * (sd[3 * j + 1] + k2x + k2z), a3 = -beta * sd[3 * j + 2];
        const double iv = 1.0 / (a2 - a1 * x);
        x = a3 * iv;
        return iv;
    };
    const bool exact = I.flag_ctpress == 0 && w.j == 0 && !v;
#pragma unroll 1
    for (int it = 0; exact && it < L; it++) {
        double e = x;
#pragma unroll 1
        for (int j = r0; j < r1; j++) pivot(j, e);
        ends[t] = e;
        __syncthreads();
        const double y = b == 0 ? x : ends[t - C];
        const bool moved = __double_as_longlong(x) != __double_as_longlong(y);
        x = y;
        if (!__syncthreads_or(moved)) break;
    }
    if (w.j * C + t % C >= nc) return;
    double *inv = (v ? I.FACV : I.FACU) + col;
#pragma unroll 1
    for (int j = r0; j < r1; j++) inv[(size_t)j * nc] = pivot(j, x);
    if (r0 <= n && r1 == n + 1) inv[(size_t)(n + 1) * nc] = 1.0 / (1.0 - wt * x);
}

__device__ __forceinline__ void cp8(void *s, const void *g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g));
}

template <int C>
__global__ void __launch_bounds__(kTileBlocks *C, 8 / C) k_column_tile(const Inst *__restrict__ insts,
                                                              const Work *__restrict__ work, int kRK)
{
    constexpr int L = kTileBlocks, T = L * C;
    extern __shared__ double2 tile_mem[];
    const Work w = work[blockIdx.x];
    const Inst &I = insts[w.inst];
    const int t = threadIdx.x, c = t % C, b = t / C;
    const int nc = I.nc, nxh = I.nxh, nyu = I.nyu, nyv = I.nyv, R = nyu + 1;
    const int col = w.j * C + c;
    const bool live = col < nc;            // lanes past the last column compute on it and store nothing
    const int cc = live ? col : nc - 1;

    // rows 1..nyu of each field at (row - 1) * C, row 0 of S2 (zero) below it
    double2 *S1 = tile_mem + c, *S3 = S1 + (size_t)nyu * C, *S2 = S3 + (size_t)R * C, *PS = S2 + (size_t)R * C;
    double *invu = reinterpret_cast<double *>(PS - c) + c, *invv = invu + (size_t)nyu * C;
    double *SG2 = reinterpret_cast<double *>(PS - c + (size_t)R * C) + c, *SG3 = SG2 + (size_t)nyu * C;
    double *scan = SG3 - c + (size_t)nyu * C;
    double *du = scan + tile_scan_doubles(C), *dv = du + 3 * (R + 1), *thu = dv + 3 * (R + 1), *thv = thu + R + 1, *dg1 = thv + R + 1;

    const int i = cc % nxh, kr = cc / nxh;
    const RK rk = rk_coeffs(kRK);
    const double dt = I.sc[SC_DT], Re = I.Re, ddv = I.ddthetavi;
    const double kxr = I.kx[i], kzr = I.kz[kr], k2 = I.k2x[i] + I.k2z[kr];
    const double beta = rk.b * dt / Re;
    const bool mean = cc == 0;
    const bool exact = I.flag_ctpress == 0 && w.j == 0;  // this tile holds the mean mode of a constant-flow-rate run
    const double2 zero = make_double2(0.0, 0.0);
    const int K = (nyu + L - 1) / L, q0 = min(nyu + 1, 1 + b * K), q1 = min(nyu + 1, q0 + K);  // rows of this lane

    // ---- 2: right-hand sides, elimination and back substitution -------------------
    // Interior rows 1..n of the systems: rows 0 contribute y = 0; the top row of
    // the u grid is the map that starts the back substitution, the v grid's is
    // zero.  u2 has no row nyu: its pivot there is taken as 0, which makes it 0.
    Aff<3> m;
    m.reset();
    {
        const double C1 = rk.a / Re, C2 = -rk.c, G = -rk.g, C3x = rk.d * kxr, C3z = rk.d * kzr;
        const double C1m = mean ? -rk.d * I.sc[SC_MPGX] : 0.0;
        // every field as a 32-bit offset from U1 (the instance is one block)
        double2 *const B = I.U1;
        const unsigned at = (unsigned)min(q0, nyu) * nc + cc;  // row q0
        const unsigned U3 = I.U3 - B, U2 = I.U2 - B, P = I.P - B, FU = I.UVF - B, FW = I.WVF - B, FV = I.VVC - B;
        const unsigned N1 = I.NU1 - B - nc, N3 = I.NU3 - B - nc, N2 = I.NU2 - B - nc;
        const unsigned X1 = I.NXZ1 - B - nc, X3 = I.NXZ3 - B - nc, X2 = I.NXZ2 - B - nc;
        unsigned o = at;
        // the rows go through the read-only path: a CTA reads only its own
        // columns here, before any of its writes
        auto ld = [&](unsigned f) { return __ldg(B + (f + o)); };
        double2 um1 = ld(-nc), uc1 = ld(0), um3 = ld(U3 - nc), uc3 = ld(U3), um2 = ld(U2 - nc), uc2 = ld(U2),
                f1 = ld(FU - nc), f3 = ld(FW - nc), f2 = ld(FV), p = ld(P - nc);
        struct Row {
            double2 up1, up3, up2, pn, no1, no3, no2, x1, x3, x2, g1, g3, g2;
        };
        auto load = [&](int j) {
            Row r;
            const bool top = j >= nyu;
            r.up1 = ld(nc), r.up3 = ld(U3 + nc), r.up2 = top ? zero : ld(U2 + nc), r.pn = top ? zero : ld(P);
            r.no1 = kRK != 1 ? ld(N1) : zero, r.no3 = kRK != 1 ? ld(N3) : zero,
            r.no2 = kRK != 1 ? ld(N2) : zero;  // c_1 = 0: Nu_old unused
            r.x1 = ld(X1), r.x3 = ld(X3), r.x2 = ld(X2), r.g1 = ld(FU), r.g3 = ld(FW), r.g2 = ld(FV + nc);
            return r;
        };
        Row ra = load(q0);
        // pivots, DG factors and y metrics to shared memory, the first row in flight
        for (int j = b; j < nyu; j += L) {
            const size_t o = (size_t)j * nc + cc;
            cp8(invu + j * C, I.FACU + o + nc);
            cp8(invv + j * C, I.FACV + o + nc);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        for (int j = b; j < nyu; j += L) {
            const size_t o = (size_t)j * nc + cc;
            cp8(SG2 + j * C, I.DG2 + o);
            cp8(SG3 + j * C, I.DG3 + o);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        for (int j = t; j <= nyu; j += T) {
            du[3 * j] = I.dyu2i[3 * j];
            du[3 * j + 1] = I.dyu2i[3 * j + 1];
            du[3 * j + 2] = I.dyu2i[3 * j + 2];
            thu[j] = I.dthdyu[j];
            dv[3 * j] = I.dyv2i[3 * j];
            dv[3 * j + 1] = I.dyv2i[3 * j + 1];
            dv[3 * j + 2] = I.dyv2i[3 * j + 2];
            thv[j] = I.dthdyv[j];
            dg1[j] = I.DG1[j];
        }
        if (t < C) S2[-C] = make_double2(0.0, 0.0);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        auto row = [&](int j, const Row &r, unsigned o) {
            const bool top = j == nyu;
            const double2 up1 = r.up1, up3 = r.up3, up2 = r.up2, pn = r.pn, no1 = r.no1, no3 = r.no3, no2 = r.no2,
                          x1 = r.x1, x3 = r.x3, x2 = r.x2, g1 = r.g1, g3 = r.g3, g2 = r.g2;
            const double d1 = du[3 * j], d2 = du[3 * j + 1], d3 = du[3 * j + 2], mt = thu[j];
            const double cen = k2 + d2, iv = invu[(j - 1) * C], a1 = j == 1 ? 0.0 : -beta * d1;
            // C3 = -dRK*k1F: (-0, -(d k)); C3*p = ((d k) p.im, -((d k) p.re))
            auto side = [&](double2 um, double2 uc, double2 up, double2 no, double2 x, double2 g, double2 f, double C3,
                            double cm, unsigned N, double2 *S, double2 &A) {
                const double2 Lp = make_double2(d1 * um.x + cen * uc.x + d3 * up.x, d1 * um.y + cen * uc.y + d3 * up.y);
                double2 dd = make_double2(C1 * Lp.x + C2 * no.x + C3 * p.y + cm, C1 * Lp.y + C2 * no.y + -(C3 * p.x));
                const double2 nu = make_double2(x.x + (g.x - f.x) * mt * ddv, x.y + (g.y - f.y) * mt * ddv);
                if (live) B[N + o] = nu;
                dd = make_double2(dd.x + G * nu.x, dd.y + G * nu.y);
                const double2 rh = make_double2(uc.x + dt * dd.x, uc.y + dt * dd.y);
                A = make_double2((rh.x - a1 * A.x) * iv, (rh.y - a1 * A.y) * iv);
                S[(j - 1) * C] = rh;
            };
            side(um1, uc1, up1, no1, x1, g1, f1, C3x, C1m, N1, S1, m.A[0]);
            side(um3, uc3, up3, no3, x3, g3, f3, C3z, 0.0, N3, S3, m.A[1]);
            m.B[0] = -(a1 * iv) * m.B[0];
            um1 = uc1, uc1 = up1, f1 = g1;
            um3 = uc3, uc3 = up3, f3 = g3;
            const double e1 = dv[3 * j], e2 = dv[3 * j + 1], e3 = dv[3 * j + 2], mv = thv[j];
            const double cenv = k2 + e2, ivv = top ? 0.0 : invv[(j - 1) * C], b1 = j == 1 ? 0.0 : -beta * e1;
            const double2 Lp = make_double2(e1 * um2.x + cenv * uc2.x + e3 * up2.x, e1 * um2.y + cenv * uc2.y + e3 * up2.y);
            const double C3 = -rk.d * ddv * mv;
            double2 dd = make_double2(C1 * Lp.x + C2 * no2.x + C3 * (pn.x - p.x), C1 * Lp.y + C2 * no2.y + C3 * (pn.y - p.y));
            const double2 nu = make_double2(x2.x + (g2.x - f2.x) * mv * ddv, x2.y + (g2.y - f2.y) * mv * ddv);
            if (live && !top) B[N2 + o] = nu;
            dd = make_double2(dd.x + G * nu.x, dd.y + G * nu.y);
            const double2 rh = top ? zero : make_double2(uc2.x + dt * dd.x, uc2.y + dt * dd.y);
            m.A[2] = make_double2((rh.x - b1 * m.A[2].x) * ivv, (rh.y - b1 * m.A[2].y) * ivv);
            m.B[1] = -(b1 * ivv) * m.B[1];
            S2[(j - 1) * C] = rh;
            um2 = uc2, uc2 = up2, f2 = g2, p = pn;
        };
#pragma unroll 1
        for (int j = q0; j < q1; j += 2) {
            const unsigned oa = o;
            if (j + 1 < q1) o += nc;
            const Row rb = load(j + 1);
            row(j, ra, oa);
            const unsigned ob = o;
            if (j + 2 < q1) o += nc;
            ra = load(j + 2);
            if (j + 1 < q1) row(j + 1, rb, ob);
        }
    }
    Aff<3> *const part0 = reinterpret_cast<Aff<3> *>(scan), *const part1 = part0 + kTileBlocks / 4 * C;
    Aff<3> y = scan_entry<C, 3>(m, part0, true);
    if (exact)
        y.A[0] = exact_entries<C, true>(y.A[0], reinterpret_cast<double2 *>(scan), [&](double2 v) {
#pragma unroll 1
            for (int j = q0; j < q1; j++) {
                const double a1 = j == 1 ? 0.0 : -beta * du[3 * j], iv = invu[(j - 1) * C];
                const double2 r = S1[(j - 1) * C];
                v = make_double2((r.x - a1 * v.x) * iv, (r.y - a1 * v.y) * iv);
            }
            return v;
        });
    m.reset();
#pragma unroll 1
    for (int j = q0; j < q1; j++) {
        const int e = (j - 1) * C;
        const double iv = invu[e], a1 = j == 1 ? 0.0 : -beta * du[3 * j], f = -beta * du[3 * j + 2] * iv;
        const double ivv = j == nyu ? 0.0 : invv[e], b1 = j == 1 ? 0.0 : -beta * dv[3 * j], fv = -beta * dv[3 * j + 2] * ivv;
        const double2 r1 = S1[e], r3 = S3[e], r2 = S2[e];
        y.A[0] = make_double2((r1.x - a1 * y.A[0].x) * iv, (r1.y - a1 * y.A[0].y) * iv);
        y.A[1] = make_double2((r3.x - a1 * y.A[1].x) * iv, (r3.y - a1 * y.A[1].y) * iv);
        y.A[2] = make_double2((r2.x - b1 * y.A[2].x) * ivv, (r2.y - b1 * y.A[2].y) * ivv);
        S1[e] = y.A[0];
        S3[e] = y.A[1];
        S2[e] = y.A[2];
#pragma unroll
        for (int k = 0; k < 3; k++) m.A[k] = m.at(k, y.A[k]);
        m.B[0] = -f * m.B[0];
        m.B[1] = -fv * m.B[1];
    }
    Aff<3> u;
    u.reset();
    const bool holds_top = q0 <= nyu && q1 == nyu + 1;
    if (holds_top) {
        // the top row of u1 and u3, [gw2, 1, 0]: y = -gw2 y(nyu) inv
        const double g = __ldg(I.FACU + (size_t)(nyu + 1) * nc + cc), gw2 = I.gw2;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            u.A[k] = make_double2((0.0 - gw2 * y.A[k].x) * g, (0.0 - gw2 * y.A[k].y) * g);
            m.A[k] = m.at(k, u.A[k]);
        }
        m.B[0] = m.B[1] = 0.0;
    }
    {
        const Aff<3> in = scan_entry<C, 3>(m, part1, false);
        if (!holds_top) u = in;
    }
    if (exact) {
        const double2 v = exact_entries<C, false>(u.A[0], reinterpret_cast<double2 *>(scan), [&](double2 v) {
            if (holds_top) v = u.A[0];
#pragma unroll 1
            for (int j = q1 - 1; j >= q0; j--) {
                const double f = -beta * du[3 * j + 2] * invu[(j - 1) * C];
                const double2 r = S1[(j - 1) * C];
                v = make_double2(r.x - f * v.x, r.y - f * v.y);
            }
            return v;
        });
        if (!holds_top) u.A[0] = v;
    }
#pragma unroll 1
    for (int j = q1 - 1; j >= q0; j--) {
        const int e = (j - 1) * C;
        const double f = -beta * du[3 * j + 2] * invu[e], fv = j == nyu ? 0.0 : -beta * dv[3 * j + 2] * invv[e];
        const double2 r1 = S1[e], r3 = S3[e], r2 = S2[e];
        u.A[0] = make_double2(r1.x - f * u.A[0].x, r1.y - f * u.A[0].y);
        u.A[1] = make_double2(r3.x - f * u.A[1].x, r3.y - f * u.A[1].y);
        u.A[2] = make_double2(r2.x - fv * u.A[2].x, r2.y - fv * u.A[2].y);
        S1[e] = u.A[0];
        S3[e] = u.A[1];
        S2[e] = u.A[2];
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");  // DG
    __syncthreads();

    const double dtirk = (1.0 / dt) / (rk.a + rk.b);
    if (exact) {  // uniform in the CTA
        // flowrate_corr (littleharsh.f90:515-548) with LU_build0 (tridLU_3D.f90:
        // 299-325), whose matrix is the mean mode's: its pivots are column 0's.
        // flowrateRe's dummy u(1:nn+2) receives u11(0:nn+2), so it sums u11(j-1).
        // u11 takes the place of the v-grid pivots.
        double *u11 = invv - c, *q = scan;
        if (t == 0) {
            const double bdt = -rk.d * dt;
            double y = 0.0;
#pragma unroll 4
            for (int j = 1; j <= nyu; j++) {
                const double a1 = j == 1 ? 0.0 : -beta * du[3 * j];
                y = (bdt - a1 * y) * invu[(j - 1) * C];
                u11[j] = y;
            }
            y = (0.0 - I.gw2 * y) * I.FACU[(size_t)(nyu + 1) * nc];
#pragma unroll 4
            for (int j = nyu; j >= 1; j--) {
                y = u11[j] - -beta * du[3 * j + 2] * invu[(j - 1) * C] * y;
                u11[j] = y;
            }
            u11[0] = 0.0 - I.gw1 * y;
            double Qx1 = 0.0;
#pragma unroll 4
            for (int j = 1; j <= nyv + 1; j++) Qx1 = Qx1 + (I.yv[j] - I.yv[j - 1]) * u11[j - 1];
            q[0] = Qx1;
        } else if (t == 32) {
            double Qx0 = 0.0;
#pragma unroll 4
            for (int j = 1; j <= nyv + 1; j++) Qx0 = Qx0 + (I.yv[j] - I.yv[j - 1]) * tile_mem[(j - 1) * C].x;
            q[1] = Qx0;
        }
        __syncthreads();
        const double g = (I.sc[SC_QXT] - q[1]) / q[0];
        for (int j = 1 + t; j <= nyu; j += T) tile_mem[(j - 1) * C].x = tile_mem[(j - 1) * C].x + g * u11[j];
        if (t == 0) {
            I.sc[SC_MPGX] = I.sc[SC_MPGX] + g;
            I.sc[SC_DGX] = g;
        }
        __syncthreads();
    }

    // ---- 3: divergence, LUsolP, p += psi, v_corr ------------------------------------
    {
        Aff<1> s;
        Aff<1> *const tot0 = reinterpret_cast<Aff<1> *>(part0), *const tot1 = reinterpret_cast<Aff<1> *>(part1);
        // psi = div / (dt (a+b)); forward x_j = (ps_j - g1_j x_{j-1}) g2_j
        s.reset();
        double2 vm = S2[(q0 - 2) * C];
#pragma unroll 1
        for (int j = q0; j < q1; j++) {
            const int e = (j - 1) * C;
            const double g2 = SG2[e], g1 = j == 1 ? 0.0 : dg1[j];
            const double2 a = S1[e], c3 = S3[e], vc = S2[e];
            const double mm = ddv * thu[j];
            double2 ps = cscale(dtirk, make_double2(-(kxr * a.y) + -(kzr * c3.y) + mm * (vc.x - vm.x),
                                                    kxr * a.x + kzr * c3.x + mm * (vc.y - vm.y)));
            if (mean && j == 1) ps = zero;
            PS[e] = ps;
            s.A[0] = make_double2((ps.x - g1 * s.A[0].x) * g2, (ps.y - g1 * s.A[0].y) * g2);
            s.B[0] = -(g1 * g2) * s.B[0];
            vm = vc;
        }
        double2 x = scan_entry<C, 1>(s, tot0, true).A[0];
        s.reset();
#pragma unroll 1
        for (int j = q0; j < q1; j++) {
            const int e = (j - 1) * C;
            const double g2 = SG2[e], g1 = j == 1 ? 0.0 : dg1[j], g3 = j < nyu ? SG3[e] : 0.0;
            const double2 ps = PS[e];
            x = make_double2((ps.x - g1 * x.x) * g2, (ps.y - g1 * x.y) * g2);
            PS[e] = x;
            s.A[0] = s.at(0, x);
            s.B[0] = -g3 * s.B[0];
        }
        // back: psi_j = x_j - g3_j psi_{j+1} (g3 of the last row is zero), p +=
        // psi, v_corr (littleharsh.f90:896-993): u1 and u3 need psi(j), u2
        // psi(j) and psi(j+1)
        double2 pn = scan_entry<C, 1>(s, tot1, false).A[0];
        const double dtrk = dt * (rk.a + rk.b);
        const double kd1 = dtrk * kxr, kd3 = dtrk * kzr, dtrk_u2 = dtrk * ddv;
        double2 *U1 = I.U1 + cc, *U2 = I.U2 + cc, *U3 = I.U3 + cc, *P = I.P + cc;
        double2 pv = q0 < q1 ? P[(size_t)(q1 - 2) * nc] : zero;  // p one row ahead
#pragma unroll 1
        for (int j = q1 - 1; j >= q0; j--) {
            const size_t o = (size_t)j * nc;
            const int e = (j - 1) * C;
            const double2 pold = pv;
            if (j > q0) pv = P[o - 2 * (size_t)nc];
            double2 ps = PS[e];
            if (j < nyu) {
                const double g3 = SG3[e];
                ps = make_double2(ps.x - g3 * pn.x, ps.y - g3 * pn.y);
            }
            double2 a1 = S1[e], a3 = S3[e];
            const double2 a2 = S2[e];
            a1 = make_double2(a1.x - -(kd1 * ps.y), a1.y - kd1 * ps.x);
            a3 = make_double2(a3.x - -(kd3 * ps.y), a3.y - kd3 * ps.x);
            const double mv = dtrk_u2 * thv[j];
            if (live) {
                P[o - nc] = make_double2(pold.x + ps.x, pold.y + ps.y);
                U1[o] = a1;
                U3[o] = a3;
                U2[o] = j < nyu ? make_double2(a2.x - mv * (pn.x - ps.x), a2.y - mv * (pn.y - ps.y)) : zero;
                if (j == 1 || j == nyu) {  // ghost and wall rows
                    const size_t g = j == 1 ? 0 : o + nc;
                    const double gw = I.gwbc;
                    U1[g] = cscale(gw, a1);
                    U3[g] = cscale(gw, a3);
                    if (j == 1) {
                        U2[0] = zero;
                        if (!isfinite(a1.x) || !isfinite(a1.y) || !isfinite(a3.x) || !isfinite(a3.y) ||
                            !isfinite(ps.x) || !isfinite(ps.y))
                            atomicOr(I.err, ERR_NONFINITE);
                    }
                }
            }
            if (mean) S1[e] = a1;
            pn = ps;
        }
    }
    if (w.j == 0 && kRK == 3) {
        __syncthreads();
        if (t == 0) {
            // flowrateIm (littleharsh.f90:473-492) via meanflow_ctP (:572-589)
            double Qu = 0.0;
#pragma unroll 4
            for (int j = 1; j <= nyv + 1; j++) Qu = Qu + (I.yv[j] - I.yv[j - 1]) * tile_mem[(j - 1) * C].x;
            I.sc[SC_QX] = Qu;
            I.sc[SC_ITER] = I.sc[SC_ITER] + 1.0;
        }
    }
}

// ---------------------------------------------------------------------------
// LUsolU (tridLU_3D.f90:38-94, with LU_build + LU_dec) on plane-major columns,
// 32 lanes to a column, K rows a lane in registers, so the right-hand side is
// read once and the solution written once (in place too: a CTA has read its
// columns before it writes them).  Pivots and substitutions as in the tiles:
// composed maps, entries, then the reference's rows.  One lane a column
// (k_lusolu) waits on its loads row by row in two sweeps and keeps the factors
// in global memory in between.  Bound by HBM and, at the 8 columns of a CTA, by
// the latency of the scans: 41 MB at 128x128x153, 57 -> 21 us a call on B200.
template <int K>
__global__ void __launch_bounds__(kTileBlocks * 8) k_lusolu_tile(const Inst *__restrict__ insts, int grid, int kRK,
                                                                 double dt, const double2 *rhs, double2 *u)
{
    constexpr int C = 8, T = kTileBlocks * C;
    extern __shared__ double sd[];  // the grid's d2/dy2 coefficients
    __shared__ Mob maps[T];
    __shared__ Aff<1> part[2][kTileBlocks / 4 * C];
    const Inst &I = insts[0];
    const int t = threadIdx.x, c = t % C, b = t / C, nc = I.nc, nxh = I.nxh;
    const int n = grid == 2 ? I.nyu : I.nyv;  // rows 0..n+1
    const int col = blockIdx.x * C + c, cc = min(col, nc - 1), r0 = b * K;
    double2 r[K];
#pragma unroll
    for (int q = 0; q < K; q++) r[q] = rhs[(size_t)min(r0 + q, n + 1) * nc + cc];
    const double *d = grid == 2 ? I.dyu2i : I.dyv2i;
    for (int e = t; e < 3 * (n + 1); e += T) sd[e] = d[e];
    const double k2x = I.k2x[cc % nxh], k2z = I.k2z[cc / nxh];
    const double beta = rk_coeffs(kRK).b * dt / I.Re;
    const double w0 = grid == 2 ? I.gw1 : 0.0, wt = grid == 2 ? I.gw2 : 0.0;
    __syncthreads();
    // pivots
    Mob m{1.0, 0.0, 0.0, 1.0};
    const double sc = helm_scale(beta, sd, k2x, k2z);
#pragma unroll
    for (int q = 0; q < K; q++) {
        if (r0 + q > n + 1) continue;
        const HRow h = helm_row(r0 + q, n, sd, beta * sc, k2x, k2z, w0, wt, sc);
        m = Mob{h.a3 * m.c, h.a3 * m.d, fma(h.a2, m.c, -h.a1 * m.a), fma(h.a2, m.d, -h.a1 * m.b)};
    }
    mob_rescale(m);
    maps[t] = m;
    __syncthreads();
    double p = 0.0, s = 1.0;  // the entering scaled diagonal as p / s (row 0 ignores it)
#pragma unroll 4
    for (int k = c; k < t; k += C) {
        const Mob f = maps[k];
        const double x = fma(f.a, p, f.b * s);
        s = fma(f.c, p, f.d * s);
        p = x;
    }
    double x = p / s, iv[K];
    Aff<1> a;
    a.reset();
#pragma unroll
    for (int q = 0; q < K; q++) {
        if (r0 + q > n + 1) continue;
        const HRow h = helm_row(r0 + q, n, sd, beta, k2x, k2z, w0, wt);
        iv[q] = 1.0 / (h.a2 - h.a1 * x);
        x = h.a3 * iv[q];
        a.A[0] = make_double2((r[q].x - h.a1 * a.A[0].x) * iv[q], (r[q].y - h.a1 * a.A[0].y) * iv[q]);
        a.B[0] = -(h.a1 * iv[q]) * a.B[0];
    }
    double2 y = scan_entry<C, 1>(a, part[0], true).A[0];
    a.reset();
#pragma unroll
    for (int q = 0; q < K; q++) {
        if (r0 + q > n + 1) continue;
        const HRow h = helm_row(r0 + q, n, sd, beta, k2x, k2z, w0, wt);
        y = make_double2((r[q].x - h.a1 * y.x) * iv[q], (r[q].y - h.a1 * y.y) * iv[q]);
        r[q] = y;
        iv[q] = h.a3 * iv[q];  // the scaled upper diagonal
        a.A[0] = a.at(0, y);
        a.B[0] = -iv[q] * a.B[0];
    }
    double2 v = scan_entry<C, 1>(a, part[1], false).A[0];
#pragma unroll
    for (int q = K - 1; q >= 0; q--) {
        if (r0 + q > n + 1) continue;
        v = make_double2(r[q].x - iv[q] * v.x, r[q].y - iv[q] * v.y);
        if (col < nc) u[(size_t)(r0 + q) * nc + col] = v;
    }
}

// Loads every kernel lusolu_launch may pick on the current device, so that none
// is loaded for the first time inside a stream capture.
cudaError_t lusolu_load()
{
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, (const void *)k_lusolu_tile<5>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, (const void *)k_lusolu_tile<9>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, (const void *)k_lusolu);
    return e;
}

// LUsolU of every column; fac: scratch of rows x columns for columns too tall
// for the lanes' registers.
void lusolu_launch(const Inst *insts, int grid, int kRK, double dt, int rows, int nc, const double2 *rhs, double2 *u,
                   double *fac, cudaStream_t st)
{
    const unsigned blocks = (unsigned)((nc + 7) / 8);
    const size_t smem = 3 * (size_t)rows * sizeof(double);
    if (rows <= 5 * kTileBlocks) k_lusolu_tile<5><<<blocks, kTileBlocks * 8, smem, st>>>(insts, grid, kRK, dt, rhs, u);
    else if (rows <= 9 * kTileBlocks)
        k_lusolu_tile<9><<<blocks, kTileBlocks * 8, smem, st>>>(insts, grid, kRK, dt, rhs, u);
    else k_lusolu<<<(nc + 127) / 128, 128, 0, st>>>(insts, grid, kRK, dt, rhs, u, fac);
}

cudaError_t column_tile_attributes(int C, size_t smem)
{
    return raise_smem_limit(C == 8 ? (const void *)k_column_tile<8>
                                   : (C == 4 ? (const void *)k_column_tile<4> : (const void *)k_column_tile<2>), smem);
}

void column_tile_launch(int C, unsigned grid, size_t smem, cudaStream_t st, const Inst *insts, const Work *work, int kRK)
{
    if (C == 8) k_column_tile<8><<<grid, kTileBlocks * C, smem, st>>>(insts, work, kRK);
    else if (C == 4) k_column_tile<4><<<grid, kTileBlocks * C, smem, st>>>(insts, work, kRK);
    else k_column_tile<2><<<grid, kTileBlocks * C, smem, st>>>(insts, work, kRK);
}

void factors_launch(unsigned grid, size_t smem, cudaStream_t st, const Inst *insts, const Work *work, int kRK)
{
    k_factors<<<grid, kFactorColumns * kFactorBlocks, smem, st>>>(insts, work, kRK);
}

}  // namespace lh
