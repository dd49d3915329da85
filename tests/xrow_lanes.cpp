// The x stage of a warp (lh_xprod.cuh) on the CPU: 32 lanes as coroutines that run one
// after another from one warp-wide synchronisation to the next, in a given order.
// Between two of those the programming model leaves the order open, so spectra
// and CFL maxima must not depend on it.
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __restrict__
struct double2 {
    double x, y;
};
static double2 make_double2(double x, double y) { return double2{x, y}; }

static struct {
    int x;
} threadIdx, blockDim;
static ucontext_t g_main, g_lane[32];
static char g_stack[32][1 << 20];
static bool g_done[32];
static double g_slot[2][32];
static int g_calls[32];

static void lanes_meet() { swapcontext(&g_lane[threadIdx.x], &g_main); }
static void __syncwarp() { lanes_meet(); }
static double __shfl_sync(unsigned, double v, int src)
{
    // a value is read before its lane can come to the call after next
    const int l = threadIdx.x, k = g_calls[l]++ & 1;
    g_slot[k][l] = v;
    lanes_meet();
    return g_slot[k][src & 31];
}
static double __shfl_xor_sync(unsigned m, double v, int o) { return __shfl_sync(m, v, threadIdx.x ^ o); }
template <class T>
static T __ldg(const T *p) { return *p; }
static void __syncthreads() {}
static unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)((unsigned long long)a * b >> 32); }
static long long __double_as_longlong(double x) { return (long long)x; }
static void atomicMax(unsigned long long *, unsigned long long) {}
using std::fabs;
using std::fma;
using std::fmax;
using std::min;

#include "lh_xprod.cuh"

using namespace lh;

struct Result {
    std::vector<double2> spec;
    double m1 = 0.0, m3 = 0.0;
};

// One warp, `rows` of its RW rows present; order: the lanes from one meeting to the next.
template <int NX, bool PACKED>
struct Warp {
    using XP = XPlan<NX>;
    static constexpr int nxh = NX / 3 + 1, RW = XP::RW;
    static double2 tw[NX];
    static std::vector<double2> in, T;
    static Result out;
    static int rows;
    static double lane_m1[32], lane_m3[32];

    static void lane()
    {
        const int l = threadIdx.x;
        const bool on = l < RW * XP::N1;
        const int row0 = PACKED || !on ? 0 : l / XP::N1;
        double m1 = 0.0, m3 = 0.0;
        const int have = PACKED ? rows : (on && row0 < rows);
        xrow<NX, PACKED>(
            T.data() + (size_t)row0 * XPack<NX>::RS, tw, have, true, m1, m3,
            [&](int pair, int row, const int *k, double2 *A, double2 *B) {
                for (int q = 0; q < XP::KQ; q++) {
                    const size_t o = ((size_t)pair * RW + (PACKED ? row : row0)) * 2 * nxh + k[q];
                    A[q] = in[o];
                    B[q] = in[o + nxh];
                }
            },
            [&](int pair, int row, int k, double2 A, double2 B) {
                const size_t o = ((size_t)pair * RW + (PACKED ? row : row0)) * 2 * nxh + k;
                out.spec[o] = A;
                out.spec[o + nxh] = B;
            });
        lane_m1[l] = m1;
        lane_m3[l] = m3;
        g_done[l] = true;
        for (;;) lanes_meet();
    }

    static Result run(int present, const std::vector<int> &order)
    {
        rows = present;
        out.spec.assign((size_t)3 * RW * 2 * nxh, double2{0.0, 0.0});
        T.assign((size_t)RW * XPack<NX>::RS + NX, double2{1e3, -1e3});  // what a CTA finds in its shared memory
        for (int l = 0; l < 32; l++) {
            g_done[l] = false;
            g_calls[l] = 0;
            getcontext(&g_lane[l]);
            g_lane[l].uc_stack.ss_sp = g_stack[l];
            g_lane[l].uc_stack.ss_size = sizeof g_stack[l];
            g_lane[l].uc_link = nullptr;
            makecontext(&g_lane[l], (void (*)())lane, 0);
        }
        while (std::count(g_done, g_done + 32, true) < 32)
            for (int l : order) {
                threadIdx.x = l;
                swapcontext(&g_main, &g_lane[l]);
            }
        for (int l = 0; l < 32; l++) {
            out.m1 = fmax(out.m1, lane_m1[l]);
            out.m3 = fmax(out.m3, lane_m3[l]);
        }
        return out;
    }

    static int check()
    {
        srand(NX);
        for (int m = 0; m < NX; m++) tw[m] = double2{cos(2 * kPi * m / NX), sin(2 * kPi * m / NX)};
        in.resize((size_t)3 * RW * 2 * nxh);
        for (double2 &v : in) v = double2{rand() / (double)RAND_MAX - 0.5, rand() / (double)RAND_MAX - 0.5};
        std::vector<int> up(32), down(32), odd(32);
        for (int l = 0; l < 32; l++) {
            up[l] = l;
            down[l] = 31 - l;
            odd[l] = (l * 13 + 7) % 32;
        }
        int bad = 0;
        for (int present = 0; present <= RW; present++) {
            const Result a = run(present, up);
            double m1 = 0.0, m3 = 0.0;  // the maxima of the physical rows, term by term
            for (int row = 0; row < present; row++)
                for (int f = 0; f < 2; f++)
                    for (int x = 0; x < NX; x++) {
                        const double2 *u = in.data() + (size_t)row * 2 * nxh + f * nxh;
                        double s = u[0].x;
                        for (int k = 1; k < nxh; k++)
                            s += 2.0 * (u[k].x * tw[(size_t)k * x % NX].x - u[k].y * tw[(size_t)k * x % NX].y);
                        (f ? m3 : m1) = fmax(f ? m3 : m1, fabs(s));
                    }
            // sums of NX terms, each a few ulp
            if (fabs(a.m1 - m1) > 1e-12 * NX || fabs(a.m3 - m3) > 1e-12 * NX) {
                printf("%d packed %d rows %d: maxima %.6f %.6f, rows hold %.6f %.6f\n", NX, PACKED, present, a.m1, a.m3, m1, m3);
                bad++;
            }
            for (const auto &o : {down, odd}) {
                const Result b = run(present, o);
                if (a.m1 != b.m1 || a.m3 != b.m3 ||
                    memcmp(a.spec.data(), b.spec.data(), a.spec.size() * sizeof(double2)) != 0) {
                    printf("%d packed %d rows %d: another order of the lanes, another result\n", NX, PACKED, present);
                    bad++;
                }
            }
        }
        return bad;
    }
};
template <int NX, bool P> double2 Warp<NX, P>::tw[NX];
template <int NX, bool P> std::vector<double2> Warp<NX, P>::in;
template <int NX, bool P> std::vector<double2> Warp<NX, P>::T;
template <int NX, bool P> Result Warp<NX, P>::out;
template <int NX, bool P> int Warp<NX, P>::rows;
template <int NX, bool P> double Warp<NX, P>::lane_m1[32];
template <int NX, bool P> double Warp<NX, P>::lane_m3[32];

int main()
{
    int bad = 0;
#define LH_CASE(N) bad += Warp<N, XPack<N>::value>::check();
    LH_FAST_SIZES(LH_CASE)
#undef LH_CASE
    bad += Warp<12, false>::check() + Warp<24, false>::check() + Warp<48, false>::check();  // the one-CTA planes
    printf(bad ? "%d failures\n" : "ok\n", bad);
    return bad != 0;
}
