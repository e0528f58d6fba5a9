// wg_kernels.h -- launchers of the kernels in wg_kernels.cu (host side).
#pragma once
#include <cuda_runtime.h>

#include "wg_device.h"

namespace wg {
// Largest block of the day-pipelined kernels (k_pipeline, k_vertical_ahead).
constexpr int kMaxBlockThreads = 512;

// Launch bounds of the day-pipelined kernels per arithmetic type: FP64 runs one
// block of up to 512 threads per SM (the single-member layout); FP32 blocks of at
// most 256 threads, three per SM, so that its registers leave room for the
// warps that hide its memory latency.
template <class R> struct Bounds;
template <> struct Bounds<double> { static constexpr int threads = 512, min_blocks = 1; };
template <> struct Bounds<float> { static constexpr int threads = 256, min_blocks = 3; };
// the ensemble's vertical-ahead kernel keeps a member's whole vertical state in
// registers: two blocks per SM, no spills
template <class R, bool ENS> struct VaBounds : Bounds<R> {};
template <> struct VaBounds<float, true> { static constexpr int threads = 256, min_blocks = 2; };
// the ensemble's wavefront kernel is bound by load latency: 64 registers, so that an
// SM holds 32 warps of it, in one block where there are states for all (the warps of a
// block share its states out among themselves: two blocks of 512 17.1 ms, one 16.5)
template <class R, bool ENS> struct PipeBounds : Bounds<R> {};
template <> struct PipeBounds<float, true> { static constexpr int threads = 1024, min_blocks = 1; };
// the single-member FP64 wavefront with vertical-balance warps in the same block: 16
// warps, four per SM sub-partition, so that a thread has 128 registers
template <class R, bool ENS, bool VAW> struct WaveBounds : PipeBounds<R, ENS> {};
template <class R> struct WaveBounds<R, false, true> { static constexpr int threads = 512, min_blocks = 1; };

// Thread-to-slot layout of the single-member wavefront: each block runs
// cell_warps warps of 32 consecutive slots plus one idle warp at warp index
// idle_warp (idle_warp < 0: plain mapping, slot i on thread i mod the grid).
struct WarpLayout {
  int cell_warps = 0;
  int idle_warp = -1;
  int va_warps = 0;    // vertical-balance warps appended to each wavefront block
  bool va_on = false;  // the wavefront launches carry the next chunk's vertical balance
  int blocks = 0;
  int threads = 0;
  int join = 1;        // ensembles: blocks of the launch shape that a wavefront block joins
};
cudaError_t upload_fastmath_tables(const unsigned long long exp2_tab[256], const ulonglong2 log2_tab[256]);
cudaError_t launch_math_eval(int fn, const double *x, const double *y, double *out, size_t n, cudaStream_t st);
cudaError_t launch_gather_forcing(const float *src, float *dst, const int32_t *cell_of_slot, int n, int ndays,
                                  cudaStream_t st);
cudaError_t launch_unf_forcing(const uint32_t *raw, float *dst, const int32_t *cell_of_slot, int n, int nd_file,
                               int d_first, int nd, cudaStream_t st, bool big_endian = true);
// Fields of the state into cell order: kind 0 doubles, 1 floats (out as doubles), 2
// int32; per values per cell ([per][states] in src, [cell][per] out) at byte offset.
struct StateRow { const void *src; size_t offset; int kind, per; };
constexpr int kStateRows = 24;
struct StateRows { int count; StateRow row[kStateRows]; };
cudaError_t launch_state_rows(const StateRows &rows, char *out, const int32_t *slot_of_cell, int n, size_t N,
                              int members, int member, cudaStream_t st);
// out[row][cell][member] = src[row][slot][member] (+ land's), rows of n * members
cudaError_t launch_rows(const double *src, const double *land, double *out, const int32_t *slot_of_cell, int n,
                        int members, size_t rows, bool no_inf, cudaStream_t st);
template <class R>
cudaError_t launch_vertical(const DevCellsT<R> &c, const DevStateT<R> &s, const DevVertT<R> &v, const DevForcing &f,
                            int doy, int fday, cudaStream_t st);
// potential evapotranspiration of the days of steps [t_b, t_e) into the ring, before
// the launches that read them
template <class R>
cudaError_t launch_pet(const DevCellsT<R> &c, const DevForcing &f, const DevRingT<R> &ring, int doy0, int fday0,
                       int ndays, int t_b, int t_e, cudaStream_t st);
template <class R>
int pipeline_max_blocks(bool fused, bool ens, int threads, bool vaw = false, bool wt = false, bool wu = false);
// blocks of k_vertical_ahead resident on the whole device at once (its own occupancy)
template <class R>
int vertical_ahead_max_blocks(bool ens, int threads);
template <class R>
cudaError_t launch_pipeline(bool fused, const DevCellsT<R> &c, const DevStateT<R> &s, const DevVertT<R> &v,
                            const DevForcing &f, const DevMembers &mem, const DevBalance &b, const DevRingT<R> &ring,
                            const DevSync &sync, double *outq, double *qst, int doy0, int fday0, int oday0, int ndays,
                            int t_b, int t_e, int blocks, int threads, const WarpLayout &lay, const DevMonthly &mon,
                            const DevVaWork &vw, const DevWaterTemp &wtp, const DevWaterUse &wu, cudaStream_t st);
cudaError_t launch_fill(double *p, size_t n, double v, cudaStream_t st);
// no outflow (and river temperature, rows_t null: none) of the cells that active leaves
// out, in nrows rows of n cells x members
cudaError_t launch_clear_skipped(double *rows, double *rows_t, const uint8_t *active, int n, int members, int nrows,
                                 cudaStream_t st);
// the outflow rows of steps [a, b) (step t in row t % nrows) into the two rows kept
// between calls (step t in row t & 1), each cell's last steps of either parity; the river
// temperature's likewise (null: none)
cudaError_t launch_keep_outflow(const double *rows, const double *rows_t, double *kept, double *kept_t,
                                const int32_t *offset, int n, int kd, int nrows, int ndays, int a, int b,
                                cudaStream_t st);
// n doubles from src to dst and, where there are any, from src_t to dst_t
cudaError_t launch_fetch_row(double *dst, const double *src, double *dst_t, const double *src_t, size_t n, cudaStream_t st);
template <class R>
cudaError_t launch_vertical_ahead(const DevCellsT<R> &c, const DevStateT<R> &s, const DevForcing &f,
                                  const DevMembers &mem, const DevBalance &b, const DevRingT<R> &ring, int doy0,
                                  int fday0, int ndays, int t_b, int t_e, int blocks, int threads, cudaStream_t st,
                                  const DevMonthly &mon, int oday0, bool dense = false);
template <class R>
cudaError_t launch_volume(const DevCellsT<R> &c, const DevStateT<R> &s, int M, double *vol, cudaStream_t st);
template <class R>
cudaError_t launch_balance_sum(const DevCellsT<R> &c, const DevStateT<R> &s, int M, const DevBalance &b,
                               const double *vol0, double *partial, int *nblocks, cudaStream_t st);
// wg_noalloc.cu: the balance sums with their scratch in a fixed device array
int64_t noalloc_max_states();
template <class R>
cudaError_t balance_noalloc(int device, const DevCellsT<R> &c, const DevStateT<R> &s, int M, const DevBalance &b,
                            const double *vol0, cudaStream_t st, double out[6]);
}  // namespace wg
