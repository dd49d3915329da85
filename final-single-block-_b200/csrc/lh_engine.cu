// Engine internals: device memory of an instance, the layout transforms at
// the host boundary, work tables and the launch sequence of a substep.
#include "lh_engine.h"

#include <cuda.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "lh_kernels.cuh"

namespace lh {

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// A kernel's dynamic shared-memory limit is process-wide and captured graphs
// of other plans may rely on it, so it is only ever raised.
cudaError_t raise_smem_limit(const void *func, size_t bytes)
{
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, func);
    if (e != cudaSuccess) return e;
    if ((size_t)fa.maxDynamicSharedSizeBytes >= bytes) return cudaSuccess;
    return cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Plane fields (Mz x nxh complex) of the staging buffer for `chunk` planes:
// the fast path's Sin (chunk + 2 kRoundStreams rows x 3 fields: the rounds in
// flight each hold a share of the chunk plus a halo row on either side) and
// Sprod (chunk x 6); the generic path uses the first 6 * chunk.
size_t staging_units(int chunk) { return (size_t)(chunk + 2 * kRoundStreams) * 3 + (size_t)chunk * kNumProducts; }

// Bytes of plane staging one chunk round may use across all instances of a
// plan, kept well inside the 126 MB L2 (LH_STAGING_MB overrides, for tuning).
// A lone instance takes up to 300 MB: its rounds' staging then spills to HBM, which the
// plane pass leaves mostly idle, but fewer launches, each of several full waves, are
// worth more.  Substep on B200, us, 96 / 150 / 200 / 300 / 500 MB: 128x128x153 357 354
// 355 351 352, 192x192x257 1502 1478 1467 1452 1442, 256x256x257 2642 2629 2616 2613
// 2604, 216x216x129 1026 975 971 971 969; an odd number of rounds loses up to 5 %.  It
// never takes more memory than lh_instance_bytes states (lone_chunk): 157 MB and 349 us
// at 128x128x153 (345 with 300), all 300 from 192x192x257 on.
// Not where the generic plane kernels run, which are slower so: 288x288x65 2408 us at
// 96 MB, 2496 at 300, 384x384x33 2133 and 2213, 288x96x65 742 and 747.
size_t staging_budget(bool lone)
{
    const char *ev = getenv("LH_STAGING_MB");
    const long mb = ev ? atol(ev) : 0;
    return (size_t)(mb > 0 ? mb : lone ? 300 : 96) << 20;
}

bool compiled_planes(const HostSetup &hs) { return fast_size(hs.Mz) && fast_size(hs.Mx); }

Tiles default_tiles(int Mx, int Mz, int nxh, int nyu, bool lone)
{
    Tiles t;
    const size_t target = 48 * 1024;
    t.bc_zinv = std::max(1, std::min(nxh, (int)(target / (32 * (size_t)Mz))));
    t.br_x = std::max(1, std::min(Mz, (int)(target / (96 * (size_t)Mx))));
    t.bc_zfwd = std::max(1, std::min(nxh, (int)(target / (192 * (size_t)Mz))));
    t.threads = 256;
    // staging capacity: the fast path holds 9 plane fields per plane plus 6
    // for the halo rows (staging_units), the generic path 6 per plane
    const size_t unit = (size_t)Mz * nxh * sizeof(double2);
    const size_t units = staging_budget(lone) / unit;
    const size_t fixed = 6 * kRoundStreams;
    t.chunk = (int)std::max<size_t>(kRoundStreams, std::min<size_t>((size_t)nyu + kRoundStreams - 1,
                                                                  units > fixed ? (units - fixed) / 9 : kRoundStreams));
    return t;
}

size_t smem_zinv(const Tiles &t, int Mz) { return 2 * (size_t)Mz * t.bc_zinv * sizeof(double2); }
size_t smem_x(const Tiles &t, int Mx) { return 2 * (size_t)Mx * 3 * t.br_x * sizeof(double2); }
size_t smem_zfwd(const Tiles &t, int Mz) { return 2 * (size_t)Mz * kNumProducts * t.bc_zfwd * sizeof(double2); }

namespace {
struct Carver {
    size_t off = 0;
    char *base = nullptr;
    template <class T>
    T *take(size_t n)
    {
        size_t o = off;
        off = align256(off + n * sizeof(T));
        return base ? reinterpret_cast<T *>(base + o) : nullptr;
    }
};

// Lay out every buffer of an instance; with base == nullptr it only sizes.  split: with
// the rows that a split column pass needs.
void carve(const HostSetup &s, int chunk, bool split, Carver &c, Inst &I, double2 **stage, size_t *stage_elems)
{
    const size_t nc = s.nc, nu = s.nyu + 2, nv = s.nyv + 2, np = s.nyu;
    I.yu = c.take<double>(nu);
    I.yv = c.take<double>(nv);
    I.dthdyu = c.take<double>(nu);
    I.dthdyv = c.take<double>(nv);
    I.dyu2i = c.take<double>(3 * nu);
    I.dyv2i = c.take<double>(3 * nv);
    I.kx = c.take<double>(s.nxh);
    I.kz = c.take<double>(s.Nz);
    I.k2x = c.take<double>(s.nxh);
    I.k2z = c.take<double>(s.Nz);
    I.DG1 = c.take<double>(s.nyu + 1);
    I.DG2 = c.take<double>(np * nc);
    I.DG3 = c.take<double>(np * nc);
    I.twz = c.take<double2>(s.Mz);
    I.twx = c.take<double2>(s.Mx);
    I.U1 = c.take<double2>(nu * nc);
    I.U2 = c.take<double2>(nv * nc);
    I.U3 = c.take<double2>(nu * nc);
    I.P = c.take<double2>(np * nc);
    I.NU1 = c.take<double2>(np * nc);
    I.NU2 = c.take<double2>(np * nc);
    I.NU3 = c.take<double2>(np * nc);
    I.NXZ1 = c.take<double2>(np * nc);
    I.NXZ2 = c.take<double2>(np * nc);
    I.NXZ3 = c.take<double2>(np * nc);
    I.UVF = c.take<double2>((np + 1) * nc);
    I.WVF = c.take<double2>((np + 1) * nc);
    I.VVC = c.take<double2>(nu * nc);
    I.FACU = c.take<double>(nu * nc);
    I.FACV = c.take<double>(nv * nc);
    I.PSI = c.take<double2>(np * nc);
    if (split) {
        I.Y1 = c.take<double2>(nu * nc);
        I.Y2 = c.take<double2>(nv * nc);
        I.Y3 = c.take<double2>(nu * nc);
        I.CARRY = c.take<double2>(18 * nc);
    }
    I.U11 = c.take<double>(nu);
    I.F11 = c.take<double>(nu);
    I.S = c.take<double2>(staging_units(chunk) * s.Mz * s.nxh);
    I.sc = c.take<double>(SC_COUNT);
    I.err = c.take<int>(8);
    *stage_elems = nu * nc;
    *stage = c.take<double2>(*stage_elems);
}
}  // namespace

size_t instance_bytes(const HostSetup &hs, int chunk, bool split)
{
    Carver c;
    Inst I{};
    double2 *st;
    size_t se;
    carve(hs, chunk, split, c, I, &st, &se);
    return c.off;
}

// A lone instance's larger staging stands where the rows of a split column pass would
// be, which only LH_COLUMN_SPLIT=1 uses: what a caller planned by lh_instance_bytes
// still fits.
int lone_chunk(const HostSetup &hs, bool compiled, bool split)
{
    const int base = default_tiles(hs.Mx, hs.Mz, hs.nxh, hs.nyu).chunk;
    if (!compiled || split) return base;
    const size_t limit = instance_bytes(hs, base, true);
    int chunk = std::max(base, default_tiles(hs.Mx, hs.Mz, hs.nxh, hs.nyu, true).chunk);
    while (chunk > base && instance_bytes(hs, chunk, false) > limit) chunk--;
    return chunk;
}

cudaError_t instance_alloc(DevInstance &d, int chunk, bool split, cudaStream_t st, void *reuse, size_t reuse_bytes)
{
    const HostSetup &s = d.hs;
    Carver c;
    Inst &I = d.inst;
    memset(&I, 0, sizeof(I));
    carve(s, chunk, split, c, I, &d.stage, &d.stage_elems);
    d.bytes = c.off;
    cudaError_t e = cudaSuccess;
    if (reuse && reuse_bytes >= d.bytes) {
        d.block = reuse;
        d.alloc_bytes = reuse_bytes;
    } else {
        e = cudaMalloc(&d.block, d.bytes);
        if (e != cudaSuccess) {
            d.block = nullptr;
            return e;
        }
        d.alloc_bytes = d.bytes;
    }
    c = Carver();
    c.base = (char *)d.block;
    carve(s, chunk, split, c, I, &d.stage, &d.stage_elems);
    e = cudaMemsetAsync(d.block, 0, d.bytes, st);
    if (e != cudaSuccess) return e;
    auto up = [&](const void *dst, const void *src, size_t bytes) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(const_cast<void *>(dst), src, bytes, cudaMemcpyHostToDevice, st);
    };
    up(I.yu, s.yu.data(), s.yu.size() * 8);
    up(I.yv, s.yv.data(), s.yv.size() * 8);
    up(I.dthdyu, s.dthdyu.data(), s.dthdyu.size() * 8);
    up(I.dthdyv, s.dthdyv.data(), s.dthdyv.size() * 8);
    up(I.dyu2i, s.dyu2i.data(), s.dyu2i.size() * 8);
    up(I.dyv2i, s.dyv2i.data(), s.dyv2i.size() * 8);
    up(I.kx, s.kx.data(), s.kx.size() * 8);
    up(I.kz, s.kz.data(), s.kz.size() * 8);
    up(I.k2x, s.k2x.data(), s.k2x.size() * 8);
    up(I.k2z, s.k2z.data(), s.k2z.size() * 8);
    up(I.DG1, s.DG1.data(), s.DG1.size() * 8);
    up(I.DG2, s.DG2.data(), s.DG2.size() * 8);
    up(I.DG3, s.DG3.data(), s.DG3.size() * 8);
    up(I.twz, s.twz.data(), s.twz.size() * 8);
    up(I.twx, s.twx.data(), s.twx.size() * 8);
    if (e != cudaSuccess) return e;
    I.Nx = s.Nx;
    I.Nz = s.Nz;
    I.Mx = s.Mx;
    I.Mz = s.Mz;
    I.nxh = s.nxh;
    I.nc = s.nc;
    I.nyu = s.nyu;
    I.nyv = s.nyv;
    I.dt_mode = d.desc.dt_mode;
    I.flag_ctpress = d.desc.flag_ctpress;
    I.nradz = (int)s.radz.size();
    I.nradx = (int)s.radx.size();
    for (int k = 0; k < I.nradz; k++) I.radz[k] = s.radz[k];
    for (int k = 0; k < I.nradx; k++) I.radx[k] = s.radx[k];
    I.Re = d.desc.Re;
    I.alp = d.desc.alp;
    I.bet = d.desc.bet;
    I.CFL = d.desc.CFL;
    I.dtv = s.dtv;
    I.dt_fixed = d.desc.dt;
    I.gw1 = s.gw1;
    I.gw2 = s.gw2;
    I.gwbc = s.gwbc;
    I.gwi1 = s.gwi1;
    I.gwi2 = s.gwi2;
    I.ddthetavi = s.ddthetavi;
    I.chunk = chunk;
    return cudaStreamSynchronize(st);
}

void instance_free(DevInstance &d)
{
    if (d.block) cudaFree(d.block);
    d.block = nullptr;
}

// Transfers of at most this many bytes between page-locked host buffers and the
// device are one kernel that reads or writes the host buffers itself instead of a
// copy and a transform per field through the staging field.  Two transfers of four
// fields on B200, copies / kernel, us: 136 columns x 98 rows (0.9 MB) up 56 / 26,
// down 54 / 25; 528 x 154 (5 MB) 134 / 116, 146 / 111; 2080 x 154 (20 MB) 428 / 431,
// 415 / 410; 8256 x 154 (81 MB) 1542 / 1684, 1486 / 1660, where the copy engine's
// larger packets win.
constexpr size_t kDirectBytes = (size_t)16 << 20;

// Whether the device may access [p, p + bytes) of host memory in place: one
// page-locked allocation or registration that holds all of it, visible under the
// same address, aligned for double2 accesses and not read-only or device I/O.
static bool direct_host(const void *p, size_t bytes)
{
    using GetAttribute = CUresult (*)(void *, CUpointer_attribute, CUdeviceptr);
    static const GetAttribute get = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return (GetAttribute)f;
    }();
    cudaPointerAttributes a;
    unsigned flags = 0;
    CUdeviceptr start = 0;
    size_t size = 0;
    if (!get || ((uintptr_t)p & 15) != 0) return false;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a.type != cudaMemoryTypeHost || a.devicePointer != p) return false;
    if (cudaHostGetFlags(&flags, const_cast<void *>(p)) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (flags & (cudaHostRegisterIoMemory | cudaHostRegisterReadOnly)) return false;
    if (get(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, (CUdeviceptr)p) != CUDA_SUCCESS ||
        get(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, (CUdeviceptr)p) != CUDA_SUCCESS)
        return false;
    return (CUdeviceptr)p >= start && (CUdeviceptr)p + bytes <= start + size;
}

// The host side of n fields (null entries move nothing); fields that share memory
// are left to the copies, which keep their order.
static bool direct_transfer(const void *const *host, const int *len, int n, int nc)
{
    size_t total = 0;
    for (int k = 0; k < n; k++) total += host[k] ? (size_t)len[k] * nc * sizeof(double2) : 0;
    if (total > kDirectBytes) return false;
    for (int k = 0; k < n; k++) {
        const size_t bk = (size_t)len[k] * nc * sizeof(double2);
        if (!host[k]) continue;
        for (int q = 0; q < k; q++) {
            const size_t bq = (size_t)len[q] * nc * sizeof(double2);
            if (host[q] && (uintptr_t)host[k] < (uintptr_t)host[q] + bq && (uintptr_t)host[q] < (uintptr_t)host[k] + bk)
                return false;
        }
        if (!direct_host(host[k], bk)) return false;
    }
    return true;
}

static cudaError_t upload_fields(DevInstance &d, const double *const *src, double2 *const *dst, const int *len, int n,
                                 cudaStream_t st)
{
    const int nc = d.hs.nc;
    const bool direct = direct_transfer((const void *const *)src, len, n, nc);
    FieldSet f;
    f.nc = nc;
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < n && e == cudaSuccess; k++) {
        const int q = direct ? k : 0;
        f.src[q] = direct ? (const double2 *)src[k] : d.stage;
        f.dst[q] = dst[k];
        f.len[q] = len[k];
        if (direct) continue;
        const size_t bytes = (size_t)len[k] * nc * sizeof(double2);
        if (!src[k]) {
            e = cudaMemsetAsync(dst[k], 0, bytes, st);
        } else {
            e = cudaMemcpyAsync(d.stage, src[k], bytes, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cols_to_planes(f, 1, st);
        }
    }
    if (direct) e = cols_to_planes(f, n, st);
    return e;
}

// Page faults of a pageable buffer that a copy is about to fill, in one call: one by
// one inside the copy they cost more than the copy itself (lh_download_state into
// fresh memory, 26 MB 12.6 -> 8.1 ms, 82 MB 40 -> 25 ms).  Whole pages inside the buffer
// only; left to the copy where four pages across the buffer are there already
// (walking those takes a tenth of their copy) and where the kernel lacks the call.
void prefault(void *p, size_t bytes)
{
#ifdef MADV_POPULATE_WRITE
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const uintptr_t a = ((uintptr_t)p + page - 1) / page * page, b = ((uintptr_t)p + bytes) / page * page;
    if (b <= a || b - a < 16 * page) return;
    bool there = true;
    for (int k = 0; k < 4 && there; k++) {
        unsigned char v = 0;
        const uintptr_t q = a + (b - a - page) / page * k / 3 * page;
        there = mincore((void *)q, page, &v) == 0 && (v & 1);
    }
    if (there) return;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) cudaGetLastError();
    else if (at.type == cudaMemoryTypeUnregistered) madvise((void *)a, b - a, MADV_POPULATE_WRITE);
#endif
}

cudaError_t download_field(const DevInstance &d, const double2 *src, int len, double *dst, cudaStream_t st)
{
    FieldSet f;
    f.nc = d.hs.nc;
    f.src[0] = src;
    f.dst[0] = d.stage;
    f.len[0] = len;
    cudaError_t e = planes_to_cols(f, 1, st);
    if (e != cudaSuccess) return e;
    const size_t bytes = (size_t)len * f.nc * sizeof(double2);
    prefault(dst, bytes);
    return cudaMemcpyAsync(dst, d.stage, bytes, cudaMemcpyDeviceToHost, st);
}

// The Nu reset and the scalars of an upload (getini).
static cudaError_t upload_scalars(DevInstance &d, const double *u1, cudaStream_t st)
{
    const HostSetup &s = d.hs;
    Inst &I = d.inst;
    StateReset r{I.NU1, I.NU2, I.NU3, (size_t)s.nyu * s.nc, I.sc, I.err, {0}};
    r.value[SC_T] = 0.0;
    r.value[SC_DT] = d.desc.dt_mode == LH_DT_FIXED ? d.desc.dt : 0.0;
    r.value[SC_MPGX] = d.desc.mpgx;
    const double q = u1 ? flowrate_host(s, u1) : 0.0;
    r.value[SC_QX] = q;
    r.value[SC_QXT] = q;  // getini: QxT = Qx for the constant flow-rate mode
    return reset_state(r, st);
}

cudaError_t instance_upload(DevInstance &d, const double *u1, const double *u2, const double *u3, const double *p,
                            cudaStream_t st)
{
    const HostSetup &s = d.hs;
    const double *src[4] = {u1, u2, u3, p};
    double2 *dst[4] = {d.inst.U1, d.inst.U2, d.inst.U3, d.inst.P};
    const int len[4] = {s.nyu + 2, s.nyv + 2, s.nyu + 2, s.nyu};
    cudaError_t e = upload_scalars(d, u1, st);
    if (e == cudaSuccess) e = upload_fields(d, src, dst, len, 4, st);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(st);
}

cudaError_t instance_upload_p_last(DevInstance &d, const double *u1, const double *u2, const double *u3,
                                   const double *p, cudaStream_t st, cudaEvent_t ev_u)
{
    const HostSetup &s = d.hs;
    const double *src[4] = {u1, u2, u3, p};
    double2 *dst[4] = {d.inst.U1, d.inst.U2, d.inst.U3, d.inst.P};
    const int len[4] = {s.nyu + 2, s.nyv + 2, s.nyu + 2, s.nyu};
    cudaError_t e = upload_scalars(d, u1, st);
    if (e == cudaSuccess) e = upload_fields(d, src, dst, len, 3, st);
    if (e == cudaSuccess) e = cudaEventRecord(ev_u, st);
    if (e == cudaSuccess) e = upload_fields(d, src + 3, dst + 3, len + 3, 1, st);
    return e;
}

cudaError_t instance_download(DevInstance &d, double *u1, double *u2, double *u3, double *p, cudaStream_t st)
{
    const HostSetup &s = d.hs;
    const Inst &I = d.inst;
    const double2 *src[4] = {I.U1, I.U2, I.U3, I.P};
    double *dst[4] = {u1, u2, u3, p};
    const int len[4] = {s.nyu + 2, s.nyv + 2, s.nyu + 2, s.nyu};
    cudaError_t e = cudaSuccess;
    if (direct_transfer((const void *const *)dst, len, 4, s.nc)) {
        FieldSet f;
        f.nc = s.nc;
        int n = 0;
        for (int k = 0; k < 4; k++) {
            if (!dst[k]) continue;
            f.src[n] = src[k];
            f.dst[n] = (double2 *)dst[k];
            f.len[n++] = len[k];
        }
        if (n) e = planes_to_cols(f, n, st);
    } else {
        for (int k = 0; k < 4 && e == cudaSuccess; k++)
            if (dst[k]) e = download_field(d, src[k], len[k], dst[k], st);
    }
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(st);
}

// Whether the sequential column pass is split into forward-sweep chunks
// beside the plane rounds (LH_COLUMN_SPLIT=0/1 overrides).
constexpr bool kColumnSplitDefault = false;
bool column_split_wanted()
{
    const char *cs = getenv("LH_COLUMN_SPLIT");
    return cs ? cs[0] == '1' : kColumnSplitDefault;
}

// Lone instances of at most this many columns x rows run the plane pass in one
// round (plan_build).
constexpr long kOneRoundRows = 60000;

// Plans of at most this many columns in all run the column pass on tiles
// (LH_SMALL_COLUMNS overrides): an SM takes 8 columns at a time, so 1184 are one
// wave of about 5 + 4.5 rows/32 us, against 0.6 us a row of k_column, whatever
// its columns: three waves from 64 rows on, two below.  Substep on B200, us,
// k_column / tiles: 2112 columns x 44 rows 53 / 53.5, 2664 x 44 60 / 71; 2664 x 97
// 119 / 115, x 153 175 / 157, x 257 285 / 251; 4704 x 97 150 / 169, x 153 229 / 239,
// x 257 384 / 381; 28 channels of 144 x 97 185 / 204.
static long tile_columns(int max_nyu) { return (max_nyu < 64 ? 2 : 3) * 1184L; }

// ---------------------------------------------------------------------------
namespace {
struct ClassTiles {
    bool fast;
    bool small = false;  // one CTA per plane (k_plane_small): a single stage, no staging
    int cbz, rbx, cbf;
    int tz, tx, tf;
    size_t smz, smx, smf;
};

// Fast-path launch shapes from upper bounds on the x modes per z-inverse
// CTA, the z rows per x CTA and the x modes per z-forward CTA; every bound is
// lowered until the block fits the kernel's launch bounds and 110 KB of
// shared memory, and the x-mode blocks are balanced.
ClassTiles fast_tiles(const HostSetup &s, int cbz_max, int rb, int cbf_max)
{
    ClassTiles c{};
    c.fast = true;
    const size_t smax = 110 * 1024;
    auto fits = [&](int stage, int M, int vectors, int per) {
        return fast_threads(M, vectors) <= fast_max_threads(stage) && (size_t)M * per * 16 <= smax;
    };
    cbz_max = std::max(1, std::min(cbz_max, s.nxh));
    while (cbz_max > 1 && !fits(0, s.Mz, cbz_max, cbz_max)) cbz_max--;
    int nb = (s.nxh + cbz_max - 1) / cbz_max;
    c.cbz = (s.nxh + nb - 1) / nb;
    c.tz = fast_threads(s.Mz, c.cbz);
    c.smz = zinv_smem(s.Mz, c.cbz);
    c.rbx = xprod_rows(s.Mx, std::max(1, std::min(rb, s.Mz)));
    c.tx = xprod_threads(s.Mx, c.rbx);
    c.smx = xprod_smem(s.Mx, c.rbx);
    cbf_max = std::max(1, std::min(cbf_max, s.nxh));
    // z forward: one half of the six products (3 vectors per x mode) per CTA
    while (cbf_max > 1 && !(zfwd_threads(s.Mz, cbf_max) <= fast_max_threads(2) && zfwd_smem(s.Mz, cbf_max) <= smax))
        cbf_max--;
    nb = (s.nxh + cbf_max - 1) / cbf_max;
    c.cbf = (s.nxh + nb - 1) / nb;
    c.tf = zfwd_threads(s.Mz, c.cbf);
    c.smf = zfwd_smem(s.Mz, c.cbf);
    return c;
}

// Default tile bounds of a fast size: measured on B200 at 128^2 (16 threads
// per vector): 16 x modes per z-inverse CTA, up to 4 x modes per z-forward CTA;
// sizes with fewer threads per vector take proportionally more.  The z-forward
// bound is 80/vz, one less at Mz = 96 and 192 (ny = 153 sweeps: one x mode fewer
// was faster there, slower at Mz = 288 and 384, even at 48).  The x stage takes
// whole CTAs of four warps; 2 to 32 rows per CTA made no difference.
void default_bounds(const HostSetup &s, int &cbz, int &rbx, int &cbf)
{
    const int vz = std::max(1, fast_vector_threads(s.Mz));
    cbz = 256 / vz;
    rbx = xprod_rows(s.Mx, s.Mz);
    cbf = std::max(1, 80 / vz - ((s.Mz == 96 || s.Mz == 192) ? 1 : 0));
}

// Tile bounds of a class: the autotuner's candidate, else the environment
// override LH_TILES=cbz,rbx,cbf, else the tuned table, else the defaults.
ClassTiles class_tiles(const HostSetup &s, bool force_generic, const TuneParams *force)
{
    ClassTiles c{};
    c.fast = !force_generic && compiled_planes(s);
    if (c.fast) {
        int a = 0, b = 0, d = 0;
        default_bounds(s, a, b, d);
        TuneParams tp;
        const char *ov = getenv("LH_TILES");
        int oa = 0, ob = 0, od = 0;
        if (force && force->cbz > 0) {
            a = force->cbz;
            b = force->rbx;
            d = force->cbf;
        } else if (ov && sscanf(ov, "%d,%d,%d", &oa, &ob, &od) == 3 && oa > 0 && ob > 0 && od > 0) {
            a = oa;
            b = ob;
            d = od;
        } else if (tune_lookup(s.Mz, s.Mx, s.nyu, tp) && tp.cbz > 0) {
            a = tp.cbz;
            b = tp.rbx;
            d = tp.cbf;
        }
        c = fast_tiles(s, a, b, d);
    } else {
        Tiles t = default_tiles(s.Mx, s.Mz, s.nxh, s.nyu);
        c.cbz = t.bc_zinv;
        c.rbx = t.br_x;
        c.cbf = t.bc_zfwd;
        c.tz = c.tx = c.tf = t.threads;
        c.smz = smem_zinv(t, s.Mz);
        c.smx = smem_x(t, s.Mx);
        c.smf = smem_zfwd(t, s.Mz);
    }
    return c;
}
}  // namespace

TuneParams default_params(const HostSetup &s)
{
    TuneParams t;
    if (compiled_planes(s)) default_bounds(s, t.cbz, t.rbx, t.cbf);
    t.staging_mb = (int)(staging_budget(compiled_planes(s)) >> 20);
    t.col_waves = 1;
    return t;
}

cudaError_t plan_build(Plan &p, const std::vector<const DevInstance *> &insts, bool force_generic,
                       const TuneParams *force)
{
    // the work buffer, side stream and events survive a rebuild
    p.rounds.clear();
    p.column.clear();
    p.force_generic = force_generic;
    p.ninst = (int)insts.size();
    // size classes in order of first appearance
    std::vector<std::pair<int, int>> classes;
    std::vector<int> cls_of(insts.size());
    int rounds = 0;
    for (size_t q = 0; q < insts.size(); q++) {
        const HostSetup &s = insts[q]->hs;
        std::pair<int, int> key(s.Mz, s.Mx);
        auto it = std::find(classes.begin(), classes.end(), key);
        if (it == classes.end()) {
            classes.push_back(key);
            it = classes.end() - 1;
        }
        cls_of[q] = (int)(it - classes.begin());
    }
    // Planes per round: the staging of the rounds in flight, summed over every instance
    // of the plan, stays inside the budget (for batches within L2, see staging_budget).
    const size_t ncls = classes.size();
    std::vector<ClassTiles> tiles(ncls);
    std::vector<const HostSetup *> rep(ncls, nullptr);
    for (size_t q = 0; q < insts.size(); q++)
        if (!rep[cls_of[q]]) rep[cls_of[q]] = &insts[q]->hs;
    for (size_t c = 0; c < ncls; c++) {
        tiles[c] = class_tiles(*rep[c], force_generic, force);
        long planes = 0;
        for (size_t q = 0; q < insts.size(); q++)
            if (cls_of[q] == (int)c) planes += insts[q]->hs.nyu;
        tiles[c].small = tiles[c].fast && small_plane_pays(rep[c]->Mx, rep[c]->Mz, planes);
    }
    // staging budget and column-pass launches: the candidate, else the
    // environment, else the tuned entry of a single-class plan, else defaults
    TuneParams tuned;
    const bool have_tuned = ncls == 1 && tune_lookup(rep[0]->Mz, rep[0]->Mx, rep[0]->nyu, tuned);
    const bool lone = insts.size() == 1;
    size_t l2_budget = staging_budget(lone && tiles[0].fast);
    if (force && force->staging_mb > 0) l2_budget = (size_t)force->staging_mb << 20;
    else if (!getenv("LH_STAGING_MB") && have_tuned && tuned.staging_mb > 0)  // tuned alone: a batch shares L2
        l2_budget = lone ? (size_t)tuned.staging_mb << 20 : std::min(l2_budget, (size_t)tuned.staging_mb << 20);
    std::vector<int> chunk_eff(insts.size());
    for (size_t q = 0; q < insts.size(); q++) {
        const HostSetup &s = insts[q]->hs;
        const bool fast = tiles[cls_of[q]].fast;
        const size_t unit = (size_t)s.Mz * s.nxh * sizeof(double2);
        const size_t units = l2_budget / (unit * insts.size());
        // kRoundStreams rounds are in flight (round r on stream r %
        // kRoundStreams), each with its share of the staging.  The L2 share
        // shrinks with the number of instances; below nyu/8 planes per round
        // the launch count costs more than staging spilling to HBM, so that
        // is the floor (within the allocated capacity).
        const size_t fixed = 6 * kRoundStreams;
        size_t c = fast ? (units > fixed ? (units - fixed) / 9 : kRoundStreams) : units / kNumProducts;
        c = std::max<size_t>(c / kRoundStreams, (size_t)(s.nyu + 7) / 8);
        c = std::max<size_t>(1, std::min<size_t>(c, (size_t)insts[q]->inst.chunk / kRoundStreams));
        // a small instance alone runs one round: two would only double its
        // launches (16^2 x 44 24.2 -> 22.6 us a substep, x 97 28.8 -> 27.4, 32^2 x
        // 97 34.2 -> 33.5, x 153 44.6 -> 46.1)
        if (fast && insts.size() == 1 && insts[q]->inst.chunk >= s.nyu && (long)s.nc * s.nyu <= kOneRoundRows) c = s.nyu;
        // and a larger one as many rounds on each stream, of about the same size
        if (fast && lone && c < (size_t)s.nyu) {
            const size_t n = ((s.nyu + c - 1) / c + kRoundStreams - 1) / kRoundStreams * kRoundStreams;
            c = (s.nyu + n - 1) / n;
        }
        if (tiles[cls_of[q]].small) c = s.nyu;  // no staging: one round
        chunk_eff[q] = (int)c;
        rounds = std::max(rounds, (s.nyu + chunk_eff[q] - 1) / chunk_eff[q]);
    }
    // The column pass: with few columns in the plan, tiles of columns in shared
    // memory (k_column_tile); otherwise 32 columns per CTA, one lane each
    // (k_column).
    size_t total_cols = 0;
    for (const DevInstance *d : insts) total_cols += (size_t)d->hs.nc;
    int max_nyu = 1;
    for (const DevInstance *d : insts) max_nyu = std::max(max_nyu, d->hs.nyu);
    const char *sc = getenv("LH_SMALL_COLUMNS");
    const bool tiled = (long)total_cols <= (sc ? atol(sc) : tile_columns(max_nyu));
    std::vector<int> width(insts.size(), 0);
    bool sequential = false;
    for (size_t q = 0; q < insts.size(); q++) {
        if (tiled) width[q] = column_tile_width(insts[q]->hs.nyu, insts[q]->hs.nc, total_cols);
        sequential |= width[q] == 0;
    }
    // Column blocks split over this many back-to-back launches (LH_COLUMN_WAVES):
    // fewer columns in flight keep the pass's intermediates in L2.
    const char *cw = getenv("LH_COLUMN_WAVES");
    p.col_waves = force && force->col_waves > 0 ? force->col_waves
                  : cw ? std::max(1, atoi(cw))
                  : (have_tuned && tuned.col_waves > 0 ? tuned.col_waves : 1);
    // work lists [round][stage][class]
    std::vector<std::vector<std::vector<std::vector<Work>>>> lists(
        rounds, std::vector<std::vector<std::vector<Work>>>(3, std::vector<std::vector<Work>>(ncls)));
    p.column.clear();
    for (int q = 0; q < (int)insts.size(); q++) {
        const HostSetup &s = insts[q]->hs;
        const ClassTiles &ct = tiles[cls_of[q]];
        const int chunk = chunk_eff[q];
        const int nbz = (s.nxh + ct.cbz - 1) / ct.cbz;
        const int nbx = (s.Mz + ct.rbx - 1) / ct.rbx;
        const int nbf = (s.nxh + ct.cbf - 1) / ct.cbf;
        if (ct.small) {
            for (int j = 1; j <= s.nyu; j++) lists[0][1][cls_of[q]].push_back({q, j, 0, 0, 0});
        } else if (ct.fast) {
            // round r: planes j0..j1 in staging half r%2; Sin slot sb+p holds
            // y row j0-1+p (u1/u3 on rows j0..j1+1, u2 on rows j0-1..j1),
            // Sprod slot pb+j-j0 plane j
            for (int j0 = 1, r = 0; j0 <= s.nyu; j0 += chunk, r++) {
                const int j1 = std::min(s.nyu, j0 + chunk - 1);
                const int sb = (r % kRoundStreams) * (chunk + 2), pb = (r % kRoundStreams) * chunk;
                auto &L = lists[r];
                for (int jp = j0 - 1; jp <= j1 + 1; jp++)
                    for (int f = 0; f < 3; f++) {
                        if (f < 2 ? jp < j0 : jp > j1) continue;
                        for (int b = 0; b < nbz; b++)
                            L[0][cls_of[q]].push_back({q, jp, sb + jp - j0 + 1, f * nbz + b, 0});
                    }
                for (int j = j0; j <= j1; j++) {
                    for (int b = 0; b < nbx; b++) L[1][cls_of[q]].push_back({q, j, pb + j - j0, b, sb + j - j0});
                    for (int b = 0; b < nbf; b++)
                        for (int h = 0; h < 2; h++) L[2][cls_of[q]].push_back({q, j, pb + j - j0, 2 * b + h, 0});
                }
            }
        } else {
            for (int j = 1; j <= s.nyu; j++) {
                const int r = (j - 1) / chunk, slot = (r % kRoundStreams) * chunk + (j - 1) % chunk;
                auto &L = lists[r];
                for (int f = 0; f < kNumProducts; f++)
                    for (int b = 0; b < nbz; b++) L[0][cls_of[q]].push_back({q, j, slot, f * nbz + b, 0});
                for (int b = 0; b < nbx; b++) L[1][cls_of[q]].push_back({q, j, slot, b, 0});
                for (int b = 0; b < nbf; b++) L[2][cls_of[q]].push_back({q, j, slot, b, 0});
            }
        }
        if (width[q] == 0)
            for (int b = 0; b < (s.nc + kColumnThreads - 1) / kColumnThreads; b++) p.column.push_back({q, b, 0, 0, 0});
    }
    std::vector<Work> all;
    p.rounds.assign(rounds, {});
    for (int r = 0; r < rounds; r++)
        for (int stg = 0; stg < 3; stg++)
            for (size_t c = 0; c < ncls; c++) {
                const auto &v = lists[r][stg][c];
                if (v.empty()) continue;
                Group g;
                g.stage = stg;
                g.fast = tiles[c].fast;
                g.small = tiles[c].small;
                g.Mz = classes[c].first;
                g.Mx = classes[c].second;
                g.off = all.size();
                g.count = v.size();
                g.threads = stg == 0 ? tiles[c].tz : stg == 1 ? tiles[c].tx : tiles[c].tf;
                g.smem = stg == 0 ? tiles[c].smz : stg == 1 ? tiles[c].smx : tiles[c].smf;
                g.param = stg == 0 ? tiles[c].cbz : stg == 1 ? tiles[c].rbx : tiles[c].cbf;
                g.grid = (unsigned)g.count;
                all.insert(all.end(), v.begin(), v.end());
                p.rounds[r].push_back(g);
            }
    p.off_column = all.size();
    all.insert(all.end(), p.column.begin(), p.column.end());
    p.col_tiles.clear();
    for (int C : {8, 4, 2}) {
        Plan::ColLaunch t;
        t.C = C;
        t.off = all.size();
        for (int q = 0; q < (int)insts.size(); q++) {
            if (width[q] != C) continue;
            const HostSetup &s = insts[q]->hs;
            for (int b = 0; b < (s.nc + C - 1) / C; b++) all.push_back({q, b, 0, 0, 0});
            t.smem = std::max(t.smem, column_tile_smem_bytes(s.nyu, C));
        }
        t.count = all.size() - t.off;
        if (t.count) p.col_tiles.push_back(t);
    }
    // LU factors of the tiled instances, both grids
    p.off_factors = all.size();
    for (int q = 0; q < (int)insts.size(); q++)
        if (width[q] != 0)
            for (int b = 0; b < (insts[q]->hs.nc + kFactorColumns - 1) / kFactorColumns; b++)
                for (int grid = 0; grid < 2; grid++) all.push_back({q, b, 0, grid, 0});
    p.n_factors = all.size() - p.off_factors;
    // split column pass: per round, every instance's rows of that round x its
    // column blocks; plus one chunk of all rows
    p.col_split = p.col_tiles.empty() && column_split_wanted();
    for (const DevInstance *d : insts) p.col_split &= d->inst.Y1 != nullptr;  // a lone context made without it
    p.col_a.assign(rounds, {0, 0});
    p.off_col_full = p.n_col_full = 0;
    if (p.col_split) {
        for (int r = 0; r < rounds; r++) {
            p.col_a[r].first = all.size();
            for (int q = 0; q < (int)insts.size(); q++) {
                const HostSetup &s = insts[q]->hs;
                const int j0 = 1 + r * chunk_eff[q];
                if (j0 > s.nyu) continue;
                const int j1 = std::min(s.nyu, j0 + chunk_eff[q] - 1);
                for (int b = 0; b < (s.nc + kColumnThreads - 1) / kColumnThreads; b++) all.push_back({q, b, j0, j1, 0});
            }
            p.col_a[r].second = all.size() - p.col_a[r].first;
        }
        p.off_col_full = all.size();
        for (int q = 0; q < (int)insts.size(); q++) {
            const HostSetup &s = insts[q]->hs;
            for (int b = 0; b < (s.nc + kColumnThreads - 1) / kColumnThreads; b++) all.push_back({q, b, 1, s.nyu, 0});
        }
        p.n_col_full = all.size() - p.off_col_full;
    }
    cudaError_t e = cudaSuccess;
    if (p.col_split) {
        if (!p.side_a) e = cudaStreamCreateWithFlags(&p.side_a, cudaStreamNonBlocking);
        if (e == cudaSuccess && !p.ev_a) e = cudaEventCreateWithFlags(&p.ev_a, cudaEventDisableTiming);
        while (e == cudaSuccess && p.ev_round.size() < (size_t)rounds) {
            cudaEvent_t ev = nullptr;
            e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
            if (e == cudaSuccess) p.ev_round.push_back(ev);
        }
        if (e != cudaSuccess) return e;
    }
    if (p.n_factors) {
        if (!p.side_f && rounds > 1) e = cudaStreamCreateWithFlags(&p.side_f, cudaStreamNonBlocking);
        if (e == cudaSuccess && !p.ev_f) e = cudaEventCreateWithFlags(&p.ev_f, cudaEventDisableTiming);
        if (e != cudaSuccess) return e;
    }
    if (!p.ev_fork) e = cudaEventCreateWithFlags(&p.ev_fork, cudaEventDisableTiming);
    for (int k = 0; k < kRoundStreams - 1 && e == cudaSuccess; k++) {
        if (!p.side[k]) e = cudaStreamCreateWithFlags(&p.side[k], cudaStreamNonBlocking);
        if (e == cudaSuccess && !p.ev_join[k]) e = cudaEventCreateWithFlags(&p.ev_join[k], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) return e;
    if (all.size() > p.work_cap) {
        if (p.d_work) cudaFree(p.d_work);
        p.d_work = nullptr;
        p.work_cap = 0;
        e = cudaMalloc(&p.d_work, all.size() * sizeof(Work));
        if (e != cudaSuccess) {
            p.d_work = nullptr;
            return e;
        }
        p.work_cap = all.size();
    }
    e = cudaMemcpy(p.d_work, all.data(), all.size() * sizeof(Work), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return e;
    // dynamic shared-memory limits for every kernel this plan launches
    size_t gz = 0, gx = 0, gf = 0;
    for (size_t c = 0; c < ncls; c++) {
        if (tiles[c].small) {
            if ((e = small_plane_attributes(classes[c].second, classes[c].first)) != cudaSuccess) return e;
        } else if (tiles[c].fast) {
            if ((e = fast_set_attributes(classes[c].first, classes[c].second, tiles[c].smz, tiles[c].smx,
                                         tiles[c].smf)) != cudaSuccess)
                return e;
        } else {
            gz = std::max(gz, tiles[c].smz);
            gx = std::max(gx, tiles[c].smx);
            gf = std::max(gf, tiles[c].smf);
        }
    }
    if (gz && (e = raise_smem_limit((const void *)k_zinv, gz)) != cudaSuccess) return e;
    if (gx && (e = raise_smem_limit((const void *)k_xprod, gx)) != cudaSuccess) return e;
    if (gf && (e = raise_smem_limit((const void *)k_zfwd, gf)) != cudaSuccess) return e;
    // k_factors holds the metrics of the tiled instances only, whose rows fit a tile (970
    // at most), so it stays below the 48 KB a launch may ask for without a raised limit
    int tiled_nyu = 0;
    for (size_t q = 0; q < insts.size(); q++)
        if (width[q] != 0) tiled_nyu = std::max(tiled_nyu, insts[q]->hs.nyu);
    p.sm_factors = 3 * (size_t)(tiled_nyu + 1) * sizeof(double);
    for (const Plan::ColLaunch &t : p.col_tiles)
        if ((e = column_tile_attributes(t.C, t.smem)) != cudaSuccess) return e;
    if (!sequential) return cudaSuccess;
    p.sm_col = column_smem_bytes(max_nyu);
    if ((e = raise_smem_limit((const void *)k_column_a, p.sm_col)) != cudaSuccess) return e;
    if ((e = raise_smem_limit((const void *)k_column_bcd, p.sm_col)) != cudaSuccess) return e;
    return raise_smem_limit((const void *)k_column, p.sm_col);
}

void plan_free(Plan &p)
{
    if (p.d_work) cudaFree(p.d_work);
    p.d_work = nullptr;
    p.work_cap = 0;
    if (p.ev_fork) cudaEventDestroy(p.ev_fork);
    p.ev_fork = nullptr;
    for (int k = 0; k < kRoundStreams - 1; k++) {
        if (p.ev_join[k]) cudaEventDestroy(p.ev_join[k]);
        if (p.side[k]) cudaStreamDestroy(p.side[k]);
        p.ev_join[k] = nullptr;
        p.side[k] = nullptr;
    }
    p.rounds.clear();
    for (cudaEvent_t ev : p.ev_round) cudaEventDestroy(ev);
    p.ev_round.clear();
    if (p.ev_a) cudaEventDestroy(p.ev_a);
    p.ev_a = nullptr;
    if (p.ev_f) cudaEventDestroy(p.ev_f);
    p.ev_f = nullptr;
    if (p.side_f) cudaStreamDestroy(p.side_f);
    p.side_f = nullptr;
    if (p.side_a) cudaStreamDestroy(p.side_a);
    p.side_a = nullptr;
}

static void time_begin(LaunchTimer *t, cudaStream_t st)
{
    if (t) cudaEventRecord(t->ev[0], st);
}

static cudaError_t time_end(LaunchTimer *t, int cls, cudaStream_t st)
{
    if (!t) return cudaSuccess;
    cudaEventRecord(t->ev[1], st);
    cudaError_t e = cudaEventSynchronize(t->ev[1]);
    float f = 0.f;
    cudaEventElapsedTime(&f, t->ev[0], t->ev[1]);
    t->ms[cls] += f;
    t->n[cls] += 1;
    return e;
}

cudaError_t launch_substep(const Plan &p, const Inst *d_insts, int kRK, bool cfl_any, cudaStream_t st,
                           LaunchTimer *timer, cudaEvent_t before_column)
{
    const int want_max = (kRK == 1 && cfl_any) ? 1 : 0;
    cudaError_t e = cudaSuccess;
    // a split column pass reads p in the forward-sweep chunks beside the
    // plane rounds: there the whole substep waits for before_column
    if (before_column && p.col_split) {
        if ((e = cudaStreamWaitEvent(st, before_column, cudaEventWaitExternal)) != cudaSuccess) return e;
        before_column = nullptr;
    }
    // round r on stream r % kRoundStreams (0 = st; their staging shares are
    // disjoint), forked from st after the work the plane pass depends on and
    // joined back before the work that consumes it; timed profiles keep one
    // stream
    const int nstreams = (timer == nullptr && p.side[0] != nullptr)
                             ? (int)std::min<size_t>(kRoundStreams, p.rounds.size()) : 1;
    if (nstreams > 1) {
        if ((e = cudaEventRecord(p.ev_fork, st)) != cudaSuccess) return e;
        for (int k = 0; k < nstreams - 1; k++)
            if ((e = cudaStreamWaitEvent(p.side[k], p.ev_fork, 0)) != cudaSuccess) return e;
    }
    // forward-sweep chunks beside the plane rounds (split column pass; not
    // when dt is only known after the plane pass, nor in timed profiles)
    const bool a_beside = p.col_split && !(kRK == 1 && cfl_any);
    const bool a_stream = a_beside && timer == nullptr && p.side_a != nullptr;
    if (a_stream) {
        if (nstreams <= 1 && (e = cudaEventRecord(p.ev_fork, st)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(p.side_a, p.ev_fork, 0)) != cudaSuccess) return e;
    }
    // the tiles' LU factors beside the plane pass too, unless dt is only known
    // after it
    const bool f_beside = p.n_factors && !(kRK == 1 && cfl_any) && timer == nullptr;
    if (f_beside) {
        if (nstreams <= 1 && !a_stream && (e = cudaEventRecord(p.ev_fork, st)) != cudaSuccess) return e;
        cudaStream_t sf = p.rounds.size() > 1 ? p.side_f : p.side[0];  // a lone round leaves the side stream free
        if ((e = cudaStreamWaitEvent(sf, p.ev_fork, 0)) != cudaSuccess) return e;
        factors_launch((unsigned)p.n_factors, p.sm_factors, sf, d_insts, p.d_work + p.off_factors, kRK);
        if ((e = cudaEventRecord(p.ev_f, sf)) != cudaSuccess) return e;
    }
    for (size_t ri = 0; ri < p.rounds.size(); ri++) {
        for (const Group &g : p.rounds[ri]) {
            const Work *w = p.d_work + g.off;
            const unsigned n = (unsigned)g.count;
            const int si = (int)(ri % kRoundStreams);
            cudaStream_t st0 = st;
            cudaStream_t st = (nstreams > 1 && si > 0) ? p.side[si - 1] : st0;
            time_begin(timer, st);
            if (g.small) {
                small_plane_launch(g.Mx, g.Mz, g.grid, st, d_insts, w, want_max);
            } else if (g.fast) {
                const int cnt = (int)g.count;
                if (g.stage == 0) fast_launch_zinv(g.Mz, g.grid, g.threads, g.smem, st, d_insts, w, cnt, g.param);
                else if (g.stage == 1)
                    fast_launch_xprod(g.Mx, g.grid, g.threads, g.smem, st, d_insts, w, cnt, g.param, want_max);
                else fast_launch_zfwd(g.Mz, g.grid, g.threads, g.smem, st, d_insts, w, cnt, g.param);
            } else {
                if (g.stage == 0) k_zinv<<<n, g.threads, g.smem, st>>>(d_insts, w, g.param);
                else if (g.stage == 1) k_xprod<<<n, g.threads, g.smem, st>>>(d_insts, w, g.param, want_max);
                else k_zfwd<<<n, g.threads, g.smem, st>>>(d_insts, w, g.param);
            }
            if ((e = time_end(timer, g.stage, st)) != cudaSuccess) return e;
        }
        if (a_beside && p.col_a[ri].second) {
            const int si = (int)(ri % kRoundStreams);
            cudaStream_t rs = (nstreams > 1 && si > 0) ? p.side[si - 1] : st;
            cudaStream_t as = rs;
            if (a_stream) {
                if ((e = cudaEventRecord(p.ev_round[ri], rs)) != cudaSuccess) return e;
                if ((e = cudaStreamWaitEvent(p.side_a, p.ev_round[ri], 0)) != cudaSuccess) return e;
                as = p.side_a;
            }
            time_begin(timer, as);
            k_column_a<<<(unsigned)p.col_a[ri].second, kColumnBlock, p.sm_col, as>>>(
                d_insts, p.d_work + p.col_a[ri].first, kRK);
            if ((e = time_end(timer, 4, as)) != cudaSuccess) return e;
        }
    }
    if (a_stream) {
        if ((e = cudaEventRecord(p.ev_a, p.side_a)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(st, p.ev_a, 0)) != cudaSuccess) return e;
    }
    for (int k = 0; k < nstreams - 1; k++) {
        if ((e = cudaEventRecord(p.ev_join[k], p.side[k])) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(st, p.ev_join[k], 0)) != cudaSuccess) return e;
    }
    if (kRK == 1) {
        time_begin(timer, st);
        k_dt<<<p.ninst, 256, 0, st>>>(d_insts, p.ninst);
        if ((e = time_end(timer, 3, st)) != cudaSuccess) return e;
    }
    if (before_column && (e = cudaStreamWaitEvent(st, before_column, cudaEventWaitExternal)) != cudaSuccess) return e;
    if (f_beside && (e = cudaStreamWaitEvent(st, p.ev_f, 0)) != cudaSuccess) return e;
    if (p.n_factors && !f_beside) {
        time_begin(timer, st);
        factors_launch((unsigned)p.n_factors, p.sm_factors, st, d_insts, p.d_work + p.off_factors, kRK);
        if ((e = time_end(timer, 4, st)) != cudaSuccess) return e;
    }
    time_begin(timer, st);
    if (p.col_split) {
        if (!a_beside)
            k_column_a<<<(unsigned)p.n_col_full, kColumnBlock, p.sm_col, st>>>(d_insts, p.d_work + p.off_col_full, kRK);
        k_column_bcd<<<(unsigned)p.column.size(), kColumnBlock, p.sm_col, st>>>(d_insts, p.d_work + p.off_column, kRK);
    } else {
        for (const Plan::ColLaunch &t : p.col_tiles)
            column_tile_launch(t.C, (unsigned)t.count, t.smem, st, d_insts, p.d_work + t.off, kRK);
        const size_t nb = p.column.size(), per = (nb + p.col_waves - 1) / p.col_waves;
        for (size_t b0 = 0; b0 < nb; b0 += per)
            k_column<<<(unsigned)std::min(per, nb - b0), kColumnBlock, p.sm_col, st>>>(
                d_insts, p.d_work + p.off_column + b0, kRK);
    }
    if ((e = time_end(timer, 4, st)) != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace lh
