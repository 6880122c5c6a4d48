// Host-side launchers of the kernel translation units.
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "cgli_dev.cuh"

namespace cgli {

// words per slot of SweepArgs::cellrec: record, MR (16 words: whole 16-byte
// vectors in both precisions)
constexpr int CR_N = REC_N + 5;
constexpr int CR_MR = REC_N;
static_assert(CR_N == 16, "record + MR fill 16 words");
// position of 16-byte vector u (0..7 FP64, 0..3 FP32) within the slot whose
// index in its step block is t: rotated by t so that the slots' vectors,
// read one per lane, spread over the shared-memory banks
template <typename T>
__host__ __device__ __forceinline__ int rec_vec_pos(int u, int t) {
  return sizeof(T) == 8 ? (u ^ (t & 7)) : (u ^ ((t >> 1) & 3));
}

// Wavefront geometry per arithmetic type of the passes: a CTA holds TI x rows
// of SWEEP_TJ = 32 j columns (a warp per row, a lane per column); the slots of
// a row's rings, by which the rows' loop is unrolled (even).
constexpr int SWEEP_TJ = 32;
template <typename T> struct SweepTile;
template <> struct SweepTile<double> {
  static constexpr int TI = 4, TJ = SWEEP_TJ, RING = 4;
};
template <> struct SweepTile<float> {
  static constexpr int TI = 4, TJ = SWEEP_TJ, RING = 4;
};
constexpr int CGLI_TIMEOUT_CODE = 6, CGLI_DIVERGED_CODE = 7;   // of the status word

// Buffers of the wavefront sweeps (kernels_sweep.cu), in the arithmetic type
// of the passes (double, or float for CGLI_MIXED).  A row's stream holds the
// blocks of its forward steps s = 0 .. sweep_steps - 1, 32 columns each.
struct SweepArgs {
  // per slot, CR_N consecutive words: the split-Jacobian / diagonal record
  // (REC_N) and the residual MR (5), so that the residual writes and the
  // sweep reads whole 16-byte vectors of one cell
  void *cellrec;
  void *dq;                       // per block [5][32]: forward result, then backward result (in place)
  void *met;                      // per block [9][32]: the metric terms (general grids only)
  // periodic lagged halos, [0] forward (plane ie), [1] backward (plane 3): dQ
  // in step order [column block][step][5][32] and the products formed from
  // it (k_halo_products); the records of planes 2 / ie+1 as [REC_N][j][k]
  void *halo[2], *hx[2], *hrec[2];
  // products handed between CTAs: [tile][step][5][32] along x, [row][column
  // block][k][5] along y; hand_bytes of both, contiguous from xbuf
  void *xbuf, *ybuf;
  size_t hand_bytes;
  unsigned int *ticket;           // tile ticket counters of the two passes
  unsigned long long *clock;      // [0] %globaltimer at the first pass, [1] at the update; [2] iterations run
  const int *order;               // tile visiting order
  double *drec;                   // DP-LUR: REC_N fields of coefficient records, reference layout (on first use)
  const double *Jtab, *etdytab;   // per-j metrics of a grid uniform in x and z
  int channel_metrics;            // 1: use Jtab / etdytab instead of the 3-D arrays
  int spin_limit;                 // bounded wait (polls) for a neighbouring tile
  int cluster_x;                  // wavefront CTAs per cluster along x
  template <typename T>
  __host__ __device__ __forceinline__ T *buf(void *p) const { return static_cast<T *>(p); }
};

// steps of a row's stream (a full block of columns)
__host__ __device__ __forceinline__ int sweep_steps(const Dev &d) { return d.nz + SWEEP_TJ - 1; }
// slot of cell (i, j, k) in the rows' streams
__host__ __device__ __forceinline__ long long skew_slot(const Dev &d, int i, int j, int k) {
  const int ntj = (d.ny + SWEEP_TJ - 1) / SWEEP_TJ, jl = (j - 2) % SWEEP_TJ;
  const long long stream = (long long)(i - 3) * ntj + (j - 2) / SWEEP_TJ;
  return (stream * sweep_steps(d) + (k - 2) + jl) * SWEEP_TJ + jl;
}
__host__ __device__ __forceinline__ long long skew_size(const Dev &d) {
  return (long long)d.nx * ((d.ny + SWEEP_TJ - 1) / SWEEP_TJ) * sweep_steps(d) * SWEEP_TJ;
}
// word of the first of (j, k)'s five values (SWEEP_TJ apart) in the halos
__host__ __device__ __forceinline__ long long halo_slot(const Dev &d, int j, int k) {
  const int jl = (j - 2) % SWEEP_TJ;
  return ((long long)((j - 2) / SWEEP_TJ) * sweep_steps(d) + (k - 2) + jl) * (5 * SWEEP_TJ) + jl;
}
// tiles of the wavefront in x and y
template <typename T> inline int sweep_tiles_x(int nx) { return (nx + SweepTile<T>::TI - 1) / SweepTile<T>::TI; }
inline int sweep_tiles_y(int ny) { return (ny + SWEEP_TJ - 1) / SWEEP_TJ; }

void sweep_tile_order(int ncx, int ntj, int rows, std::vector<int> &order);
// CTAs per cluster along x of the passes over nti x tiles
int sweep_cluster_x(int nti, bool mixed);
// shared-memory opt-in of the wavefront kernels (once per process and device)
cudaError_t sweep_kernel_attributes();
// a.met from the metrics of every interior cell
void launch_metric_stream(const Dev &d, const SweepArgs &a, cudaStream_t s, bool mixed);
// the four wavefront passes (two sweeps) of one inner iteration
void launch_sweeps(const Dev &d, const SweepArgs &a, cudaStream_t s, bool mixed);
// the update and norm partials after the last pass (k_update_skewed)
void launch_sweep_update(const Dev &d, const SweepArgs &a, cudaStream_t s, bool mixed);
// partial sums (blocks) the update after the wavefront passes writes
int sweep_update_blocks(const Dev &d);
// one pass of the first or the last sweep (a forward one with both passes'
// halo products)
void launch_sweep_pass(const Dev &d, const SweepArgs &a, cudaStream_t s, bool mixed, bool backward, bool last);
// DP-LUR inner solver of DPLUSGS.cpp (kernels_dplur.cu): residual, four
// Jacobi relaxations (final result in NR), update with per-block partial
// sums of the squared squared increments in d.partial (nx * ny blocks).
// Reads the per-j metric tables of sw when sw.channel_metrics is set.
void launch_dplur(const Dev &d, const SweepArgs &sw, cudaStream_t s);
// residual assembly writing MR and the first sweep's lagged halo planes
void launch_residual_fast(const Dev &d, const SweepArgs &a, cudaStream_t s, bool mixed);

// adds the per-(i, j) sums over k of Statistic.cpp:120-160 to sums
// [11][nx][ny] (U, V, W, T, UU, VV, WW, TT, UV, UT, VT)
void launch_statistics(const Dev &d, cudaStream_t s, double *sums);
// d.iJ = 1/J on every cell (0 where J = 0)
void launch_inverse_j(const Dev &d, cudaStream_t s);
// main.cpp:167-210: x halo (periodic slab only), Y, X (open slab only), Z
void launch_halo_bc(const Dev &d, cudaStream_t s);
// true (and d.ftab filled) when every face metric has the channel's form
// with a per-row etdy and J; dflag: one device int of scratch
bool check_face_tables(const Dev &d, int *dflag, cudaStream_t s);
// X_boundary_condition.cpp on an open slab (no-op on a periodic one)
void launch_bc_x(const Dev &d, cudaStream_t s);
// outlet sponge target velocity into d.scal[1] (open slab with an outlet layer)
void launch_target_u(const Dev &d, cudaStream_t s);
void launch_halo_x(const Dev &d, cudaStream_t s);
void launch_bc_y(const Dev &d, cudaStream_t s);
void launch_bc_z(const Dev &d, cudaStream_t s);
void launch_flux_x(const Dev &d, cudaStream_t s);
void launch_flux_y(const Dev &d, cudaStream_t s);
void launch_flux_z(const Dev &d, cudaStream_t s);
// Viscous_terms.cpp:260-904: vF of every interior cell (kernels_viscous.cu)
void launch_viscous(const Dev &d, cudaStream_t s);
// planes per CTA of a kernel that marches `cols` columns of nx planes
int march_chunk(int nx, int cols, int resident, int start);
// residual, sweeps and update of the reference-granularity path; leaves
// per-block partial sums of the squared increments in d.partial
void launch_dts(const Dev &d, cudaStream_t s, int update_blocks_x);
// reduces d.partial (nblocks x 5) into out[5] = sqrt(sum) * scale
void launch_norms(const Dev &d, cudaStream_t s, int nblocks, double scale, double *out);
// what an inner iteration leaves for the host
struct IterResult {
  double norm[5];
  double sweep_ms;   // device time of the wavefront passes (0: none)
  int status;        // the status word: a pass that gave up
};
// the norms from d.partial (as launch_norms), the status word and the passes'
// time of this iteration into ring[iteration % slots] (host memory); a norm
// that is not finite sets the status word, so that iterations launched behind
// this one leave the state alone
void launch_iteration_result(const Dev &d, const SweepArgs &a, cudaStream_t s, int nblocks, double scale,
                             IterResult *ring, int slots, bool timed);
// bulk mass flux (Driven_force.cpp:38-62) into out[0]; out holds 8 + 296
// doubles (per-block partial sums at out + 8)
void launch_bulk_flux(const Dev &d, cudaStream_t s, double *out);
// time-level shift over planes 2..ie+1 (main.cpp:364-386)
void launch_end_step(const Dev &d, cudaStream_t s);
// extrapolated initial guess of a step (order 1 or 2) on the interior cells
void launch_predict(const Dev &d, cudaStream_t s, int order);

// message returned by cgli_last_error() on this thread
void set_last_error(const std::string &msg);

}  // namespace cgli
