// Kernel declarations (definitions in lh_plane.cu and lh_column.cu).
#pragma once

#include "lh_core.cuh"

namespace lh {

constexpr int kColumnThreads = 32;       // columns per column-pass CTA (one lane each)
constexpr int kColumnBlock = 3 * kColumnThreads;  // three warps: the u1, u3 and u2 chains
size_t column_smem_bytes(int max_nyu);  // ring + staged y metrics
// column pass on tiles in shared memory (lh_column_tile.cu)
int column_tile_width(int nyu, int nc, size_t total);  // columns per tile of an instance, 0: not served
size_t column_tile_smem_bytes(int nyu, int C);
cudaError_t column_tile_attributes(int C, size_t smem);
void column_tile_launch(int C, unsigned grid, size_t smem, cudaStream_t st, const Inst *insts, const Work *work, int kRK);
// the tiles' inverse pivots into FACU / FACV, before column_tile_launch
constexpr int kFactorColumns = 8, kFactorBlocks = 32;  // columns and lanes per column of a k_factors CTA
void factors_launch(unsigned grid, size_t smem, cudaStream_t st, const Inst *insts, const Work *work, int kRK);

__global__ void k_zinv(const Inst *__restrict__ insts, const Work *__restrict__ work, int bc);
__global__ void k_xprod(const Inst *__restrict__ insts, const Work *__restrict__ work, int br, int want_max);
__global__ void k_zfwd(const Inst *__restrict__ insts, const Work *__restrict__ work, int bc);
__global__ void k_plane_z_inv(const Inst *__restrict__ insts, double *planes, int bc, int zero_row);
__global__ void k_plane_z_fwd(const Inst *__restrict__ insts, double *planes, int bc);
__global__ void k_plane_x_inv(const Inst *__restrict__ insts, double *planes, int br);
__global__ void k_plane_x_fwd(const Inst *__restrict__ insts, double *planes, int br);
__global__ void k_plane_zero_row(const Inst *__restrict__ insts, double *planes);

__global__ void k_column(const Inst *__restrict__ insts, const Work *__restrict__ work, int kRK);
// the column pass split: forward sweeps in row chunks, then phases B-D
__global__ void k_column_a(const Inst *__restrict__ insts, const Work *__restrict__ work, int kRK);
__global__ void k_column_bcd(const Inst *__restrict__ insts, const Work *__restrict__ work, int kRK);
__global__ void k_dt(const Inst *__restrict__ insts, int ninst);
// layout transforms at the host boundary: n fields of len[k] x nc
struct FieldSet {
    const double2 *src[4] = {nullptr, nullptr, nullptr, nullptr};
    double2 *dst[4] = {nullptr, nullptr, nullptr, nullptr};
    int len[4] = {0, 0, 0, 0};
    int nc = 0;
};
cudaError_t cols_to_planes(const FieldSet &f, int n, cudaStream_t st);
cudaError_t planes_to_cols(const FieldSet &f, int n, cudaStream_t st);
struct StateReset {
    double2 *nu1, *nu2, *nu3;
    size_t n;
    double *sc;
    int *err;
    double value[SC_COUNT];
};
cudaError_t reset_state(const StateReset &r, cudaStream_t st);
cudaError_t rows_to_cols(const double *src, double *dst, int len, int nc, cudaStream_t st);
__global__ void k_lusolu(const Inst *__restrict__ insts, int grid, int kRK, double dt, const double2 *rhs,
                         double2 *u, double *fac);
// the same without global scratch where the rows fit the lanes (lh_column_tile.cu)
void lusolu_launch(const Inst *insts, int grid, int kRK, double dt, int rows, int nc, const double2 *rhs, double2 *u,
                   double *fac, cudaStream_t st);
cudaError_t lusolu_load();
__global__ void k_lusolp(const Inst *__restrict__ insts, double2 *x);
__global__ void k_divmax(const Inst *__restrict__ insts, double *out);

// on-device spectra of flagged steps (lh_diag.cu): accumulator doubles and launch;
// the plane stats are declared in lh_engine.h
size_t spectra_doubles(int nyu, int nyv, int nc);
void launch_spectra_accumulate(const Inst *d_inst, double *sp, int nyu, int nc, cudaStream_t st);

// raise (never lower) a kernel's dynamic shared-memory limit (lh_engine.cu)
cudaError_t raise_smem_limit(const void *func, size_t bytes);

// the plane pass of a small plane in one CTA (lh_plane_small.cu)
bool small_plane(int Mx, int Mz);
bool small_plane_pays(int Mx, int Mz, long planes);
cudaError_t small_plane_attributes(int Mx, int Mz);
void small_plane_launch(int Mx, int Mz, unsigned grid, cudaStream_t st, const Inst *insts, const Work *work, int want_max);

// compile-time-sized fast path (lh_plane_fast.cu)
bool fast_size(int n);
int fast_threads(int n, int vectors);
int fast_max_threads(int stage);  // launch-bounds block size of a z stage
int fast_vector_threads(int n);   // threads per vector of a fast length
size_t zinv_smem(int n, int cb);  // shared memory of a z-inverse CTA of cb vectors
int xprod_rows(int n, int rb);     // z rows per CTA the kernel takes for a bound rb
int xprod_threads(int n, int rb);  // threads of an x-stage CTA of rb z rows
size_t xprod_smem(int n, int rb);  // shared memory of an x-stage CTA of rb z rows
int zfwd_threads(int n, int cb);   // threads of a z-forward CTA of cb x modes
size_t zfwd_smem(int n, int cb);   // shared memory of a z-forward CTA of cb x modes
cudaError_t fast_set_attributes(int Mz, int Mx, size_t smz, size_t smx, size_t smf);
void fast_launch_zinv(int Mz, unsigned grid, int threads, size_t smem, cudaStream_t st, const Inst *insts,
                      const Work *work, int count, int cb);
void fast_launch_xprod(int Mx, unsigned grid, int threads, size_t smem, cudaStream_t st, const Inst *insts,
                       const Work *work, int count, int rb, int want_max);
void fast_launch_zfwd(int Mz, unsigned grid, int threads, size_t smem, cudaStream_t st, const Inst *insts,
                      const Work *work, int count, int cb);

}  // namespace lh
