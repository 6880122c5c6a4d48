// LU-SGS forward / backward sweeps as a systolic wavefront of warps.
//
// The reference visits the cells of one x-slab hyperplane by hyperplane
// (i+j+k = m, Dual_time_stepping.cpp:983-1664), one OpenMP barrier per
// plane.  A cell's update depends only on its three upwind neighbours, so
// any order that respects that dependency graph gives the same numbers.
// Here one warp owns one x row (i) of 32 j columns, one column per lane, and
// marches along k: at step s of the forward pass lane jl handles cell
// k = 2 + s - jl.  Its k neighbour is its own previous step (registers), its
// j neighbour is the lane below at the previous step (a warp shuffle), and
// its i neighbour is the same lane of the warp of row i - 1 at the same step,
// which hands its products A.dQ over through a ring of shared-memory slots,
// one mbarrier per slot and direction.  The backward pass runs the mirror
// image, its steps visiting the forward steps in descending order.
//
// What bounds it: a pass is a chain of Nx + Ny + Nz dependent steps, and in
// the middle of the chain the HBM traffic of about 1200 active warps.  There
// is no block barrier: a warp waits only for the slot it needs next, so the
// chain runs at the latency of one warp's step (load the slot, about ten
// dependent FP64 operations, store the slot) and slower warps are absorbed
// by the rings.
// Measured (ms per forward / backward pass): 256x192x192 FP64 0.46 / 0.44,
// FP32 0.36 / 0.35 (a tile of 16x16 or 8x16 columns with one thread per column
// and a block barrier per step: 0.96 / 0.95 and 0.79 / 0.92); 64^3 FP64 0.084
// / 0.082 (0.248 / 0.242).  One CTA alone takes 0.36 us per step in FP64 (0.83
// before).
//
// A CTA holds TI = 4 rows (one warp per scheduler) of one 32-column block plus
// helper warps: XH x helpers fetch the x products of the row before the CTA's
// first one (each every XH-th step, so XH round trips to L2 are in flight; with
// two of them they set the pace of the FP32 passes), the y helper fetches the y
// products of the neighbouring column block for every row (a few lanes per
// row, each every QY-th step), the sender passes on what the last row posts.
// All post into the same rings the rows use among themselves, so the rows have
// no special cases; the slab's periodic x halo comes through the x helpers as
// well (products formed by k_halo_products).  Eight rows per CTA, two warps per
// scheduler, take 0.55 us per step: the shared-memory traffic of the steps
// (about 100 wavefronts a row) fills the load / store pipe; at 64^3 that made
// a pass 0.12 ms, at 256x192x192 0.51 / 0.49.
//
// Up to eight CTAs along x form a cluster.  Inside it the sender pushes the x
// products into the next CTA's ring with st.async, which counts the bytes on
// that slot's mbarrier; the receiving CTA arms the slot and returns the room
// (the receiver, a warp that takes an x helper's place).  That hop takes about
// 0.3 us; through L2 (clusters' ends, and everything along y) 1.2-1.5 us,
// which cost 0.10 against 0.084 ms a pass at 64^3.
//
// Storage.  Everything the sweeps read per cell -- the split-Jacobian /
// diagonal record with the residual MR, and dQ -- lives in per-row streams
// in the order the rows visit it: block (row, column block, forward step) of
// 32 slots.  A row's block of one step arrives by asynchronous copies of the
// row's own lanes, issued R steps ahead into the row's ring (only the lanes
// with a cell at that step are copied).  The residual kernel writes the
// records, the final update reads dQ; only these two touch the reference
// layout.
//
// Hand-over between CTAs.  Products cross through global buffers that hold a
// sentinel bit pattern wherever no value is waiting; the consumer polls the
// values themselves, so a hand-over needs no fence and no counter (4- and
// 8-byte stores are single-copy atomic), and puts the sentinel back once it
// has read a value, so the buffers are ready for the next pass without a
// fill.  A poll gives up after SweepArgs::spin_limit tries, or at once when
// its CTA or any other has given up (the CTA's dead flag, the status word):
// it records the timeout code in the status word and posts what it has, so
// that every warp runs to the end of the pass without waiting, computing
// values nobody will use; the ring waits inside a CTA follow the dead flag
// too (but not those on pushed products, which end with the row before them:
// push_wait).  The update kernel then leaves the state alone, the host reports
// CGLI_ETIMEOUT and refills the buffers with the sentinel.
// Clusters take tickets in the order in which the wavefront reaches them,
// where every dependency holds a smaller ticket, so a waiting CTA only ever
// waits on CTAs that are already running.
//
// The periodic x halo keeps the reference's lag: the forward pass at i = 3
// uses dQ of plane Nx+2 as it was at the start of the sweep, the backward
// pass at i = Nx+2 uses dQ of plane 3.  The backward pass of the first sweep
// writes both halos for the second sweep.  (Its dQ elsewhere is used by
// nothing: the second forward pass starts from MR, Dual_time_stepping.cpp:
// 1289-1293 with the lagged plane of :942-976; so only the halo planes of
// that pass are stored.)  After the final backward pass a separate, fully
// parallel kernel applies the primitive update of
// Dual_time_stepping.cpp:1702-1743 and accumulates the squared increments of
// the residual norms.
//
// T is the arithmetic type of the sweep (double, or float for CGLI_MIXED).
#include <algorithm>
#include <type_traits>

#include "cgli_dev.cuh"
#include "cgli_launch.h"
#include "tc_sm100.cuh"

namespace cgli {

// face-direction metrics of a cell: general (a row's nine terms per cell in
// the step-ordered metric stream), or a grid uniform in x and z (channel)
// whose only varying term is etdy(j)
struct MetricsGeneral {
  static constexpr bool kChannel = false;
};
struct MetricsChannel {
  static constexpr bool kChannel = true;
};

__device__ __forceinline__ double ld_gpu(const double *p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float ld_gpu(const float *p) {
  float v;
  asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool is_sentinel(double v) { return __double_as_longlong(v) == -1ll; }
__device__ __forceinline__ bool is_sentinel(float v) { return __float_as_int(v) == -1; }
__device__ __forceinline__ void put_sentinel(double *p) { *p = __longlong_as_double(-1ll); }
__device__ __forceinline__ void put_sentinel(float *p) { *p = __int_as_float(-1); }

// a wait on another tile has given up somewhere: this CTA's dead flag or
// the grid's status word (a trip to L2: polls look there now and then only)
__device__ __forceinline__ bool given_up(const volatile int *dead, const int *status) {
  return *dead || *(const volatile int *)status;
}
__device__ __forceinline__ void give_up(volatile int *dead, int *status) {
  atomicExch(status, CGLI_TIMEOUT_CODE);
  *dead = 1;
}

// Wait on a slot that counts pushed bytes, on the room for a push, and of the
// sender and the row before it.  These do not follow the dead flag: the other
// end always goes on (it is co-scheduled, and its own inputs come or are given
// up), every byte must have landed before the CTA ends, and a slot armed or
// filled ahead of its phase would leave the barrier's counts wrong.  The count
// bounds the wait against a failing device only.
constexpr int PUSH_POLLS = 1 << 26;
__device__ __noinline__ void push_wait_slow(uint32_t bar, uint32_t parity, volatile int *dead, int *status) {
  for (int n = 0; n < PUSH_POLLS; n++)
    if (tc::mbar_try(bar, parity)) return;
  give_up(dead, status);
}
__device__ __forceinline__ void push_wait(uint32_t bar, uint32_t parity, volatile int *dead, int *status) {
  if (!tc::mbar_try(bar, parity)) push_wait_slow(bar, parity, dead, status);
}

// a thread's 16-byte asynchronous copy into shared memory (not kept in L1)
// and the groups of such copies
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// Wait on a ring slot of this CTA (a phase completed by another of its
// warps).  Those warps wait on nothing but such slots and on polls that give
// up after the wait limit, and all of them follow the dead flag, so this
// ends with theirs; `polls` bounds it by itself as well.
__device__ __noinline__ void ring_wait_slow(uint32_t bar, uint32_t parity, int polls, volatile int *dead, int *status) {
  for (int n = 0; n < polls; n++) {
    if (tc::mbar_try(bar, parity)) return;
    if (*dead) return;
  }
  give_up(dead, status);
}
__device__ __forceinline__ void ring_wait(uint32_t bar, uint32_t parity, int polls, volatile int *dead, int *status) {
  if (!tc::mbar_try(bar, parity)) ring_wait_slow(bar, parity, polls, dead, status);
}

// REC_N record words and (mr non-null) the 5 MR words of one slot.  The
// 16-byte vectors of a slot are stored in an order rotated by the
// slot's position t in its step block (rec_vec_pos): a warp's vector loads
// of its slots (one per lane, consecutive slots 128 B (FP64) or 64 B (FP32)
// apart) then fall on distinct shared-memory banks in every phase of eight
// lanes.
__device__ __forceinline__ void load_cellrec(const double *p, int t, double rec[REC_N], double *mr) {
  // words 0..10 the record, 11..15 MR
  const double2 *q = reinterpret_cast<const double2 *>(p);
#pragma unroll
  for (int u = 0; u < 5; u++) {
    const double2 v = q[rec_vec_pos<double>(u, t)];
    rec[2 * u] = v.x;
    rec[2 * u + 1] = v.y;
  }
  const double2 a = q[rec_vec_pos<double>(5, t)];
  rec[10] = a.x;
  if (mr) {
    const double2 b = q[rec_vec_pos<double>(6, t)], c = q[rec_vec_pos<double>(7, t)];
    mr[0] = a.y; mr[1] = b.x; mr[2] = b.y; mr[3] = c.x; mr[4] = c.y;
  }
}
__device__ __forceinline__ void load_cellrec(const float *p, int t, float rec[REC_N], float *mr) {
  const float4 *q = reinterpret_cast<const float4 *>(p);
  const float4 a = q[rec_vec_pos<float>(0, t)], b = q[rec_vec_pos<float>(1, t)],
               c = q[rec_vec_pos<float>(2, t)];
  rec[0] = a.x; rec[1] = a.y; rec[2] = a.z; rec[3] = a.w;
  rec[4] = b.x; rec[5] = b.y; rec[6] = b.z; rec[7] = b.w;
  rec[8] = c.x; rec[9] = c.y; rec[10] = c.z;
  if (mr) {
    const float4 e = q[rec_vec_pos<float>(3, t)];
    mr[0] = c.w; mr[1] = e.x; mr[2] = e.y; mr[3] = e.z; mr[4] = e.w;
  }
}

// The x neighbour of the slab's first plane (forward) / last plane
// (backward) is the periodic halo plane 2 / ie+1, a copy of plane ie / 3 made
// by the Q halo exchange; its record is kept per (j, k), the lagged dQ of
// that plane in the rows' step order.  The products A+.dQ (forward,
// blockIdx.z = 0) and A-.dQ (backward, 1) are formed here once per sweep for
// every (j, k), off the wavefront's critical path, in step order for the
// rows' x helpers.  Both passes' products come from one launch: both inputs
// are known before the sweep's first pass.  The launch also resets the two
// passes' tickets and (first sweep) notes the time.
__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
template <class Met, bool BACKWARD, typename T>
__device__ __noinline__ void halo_product(const Dev &d, const SweepArgs &a, int j, int k) {
  const long long h = (long long)j * d.dj + k;
  T rn[REC_N], mx = 1, my = 0, mz = 0;
#pragma unroll
  for (int v = 0; v < REC_N; v++) rn[v] = a.buf<T>(a.hrec[BACKWARD])[v * d.di + h];
  if (!Met::kChannel) {
    const long long c = h + (BACKWARD ? (long long)(d.nx + 3) : 2LL) * d.di;
    mx = (T)d.m[0][c]; my = (T)d.m[1][c]; mz = (T)d.m[2][c];
  }
  const Split<T> An = split_from_record<T>(rn, 0, mx, my, mz);
  const long long s = halo_slot(d, j, k);
  T nh[5], o[5];
#pragma unroll
  for (int v = 0; v < 5; v++) nh[v] = a.buf<T>(a.halo[BACKWARD])[s + v * SWEEP_TJ];
  if (BACKWARD) upper_terms<T>(An, nh, o); else lower_terms<T>(An, nh, o);
#pragma unroll
  for (int v = 0; v < 5; v++) a.buf<T>(a.hx[BACKWARD])[s + v * SWEEP_TJ] = o[v];
}
template <class Met, typename T>
__global__ void k_halo_products(const __grid_constant__ Dev d, const __grid_constant__ SweepArgs a, int first) {
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    a.ticket[blockIdx.z] = 0;
    if (first && blockIdx.z == 0) a.clock[0] = globaltimer();
  }
  const int k = 2 + blockIdx.x * blockDim.x + threadIdx.x;
  if (k > d.nz + 1) return;
  if (blockIdx.z == 0) halo_product<Met, false, T>(d, a, 2 + blockIdx.y, k);
  else halo_product<Met, true, T>(d, a, 2 + blockIdx.y, k);
}

// the nine metric terms of every interior cell in step order (general grids;
// once per change of the metrics)
template <typename T>
__global__ void k_metric_stream(Dev d, T *out) {
  const int k = 2 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = 2 + blockIdx.y, i = 3 + blockIdx.z;
  if (k > d.nz + 1) return;
  const long long slot = skew_slot(d, i, j, k), c = ix(d, i, j, k);
  T *o = out + slot / SWEEP_TJ * (9 * SWEEP_TJ) + slot % SWEEP_TJ;
#pragma unroll
  for (int v = 0; v < 9; v++) o[v * SWEEP_TJ] = (T)d.m[v][c];
}
void launch_metric_stream(const Dev &d, const SweepArgs &a, cudaStream_t s, bool mixed) {
  const dim3 g((d.nz + 63) / 64, d.ny, d.nx);
  if (mixed) k_metric_stream<float><<<g, 64, 0, s>>>(d, (float *)a.met);
  else k_metric_stream<double><<<g, 64, 0, s>>>(d, (double *)a.met);
}

// a*b + c and a*b as written: the sums of products of a step are spelled out
// in these, so that their rounding does not depend on which of two products
// the compiler happens to fuse (it decides by the products' other uses, and
// the steps of the ramps and of the middle would round differently)
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// The split products of one direction for a face metric with a single
// nonzero component m on momentum component q = DIR + 1 (the channel grid:
// xi = (1,0,0), eta = (0,etdy,0), zeta = (0,0,1)): lower_terms / upper_terms
// of split_from_record with the zero entries left out.  (Forward, the x and z
// directions share the product hr n[0].)
template <typename T, int DIR, bool BACKWARD>
__device__ __forceinline__ void channel_products(const T r[REC_N], T m, const T n[5], T o[5]) {
  constexpr int q = DIR + 1;
  const T U = r[R_UX + DIR], lam = BACKWARD ? -r[R_LX + DIR] : r[R_LX + DIR], beta = r[R_BETA];
  const T sign = BACKWARD ? (T)1 : (T)-1;
  const T p1q = sign * mul_rn(r[R_H], m), pq1 = sign * mul_rn(r[R_HR], m), p5q = sign * mul_rn(rec_hbt<T>(r), m);
  const T p51 = sign * mul_rn(rec_g<T>(r), U);
  const T p11 = sign * mul_rn((T)0.5, fma_rn(beta, U, lam)), p22 = sign * mul_rn((T)0.5, U + lam);
  o[0] = fma_rn(p11, n[0], mul_rn(p1q, n[q]));
#pragma unroll
  for (int v = 1; v <= 3; v++)
    o[v] = v != q ? mul_rn(p22, n[v])
           : !BACKWARD && DIR != 1 ? fma_rn(p22, n[v], mul_rn(pq1, n[0]))
                                   : fma_rn(pq1, n[0], mul_rn(p22, n[v]));
  o[4] = fma_rn(p22, n[4], fma_rn(p51, n[0], mul_rn(p5q, n[q])));
}

// Geometry of a pass: TI row warps, XH x helpers, the sender and the y helper
// per CTA.
// R: slots of a row's rings (x products, y products, records), so steps of
// records on their way into shared memory.
constexpr int SWEEP_XH = 3;
template <typename T, bool GEN, bool BACKWARD>
struct SweepShape {
  static constexpr int TI = SweepTile<T>::TI, TJ = SWEEP_TJ;
  static constexpr int R = SweepTile<T>::RING;
  static constexpr int THREADS = 32 * (TI + SWEEP_XH + 2);
  static constexpr int QY = 32 / TI < R ? 32 / TI : R;   // y helper lanes per row
  // words of one ring stage: 32 slots, the forward result (backward pass),
  // the metric terms (general grids)
  static constexpr int REC = TJ * CR_N, DQ = BACKWARD ? TJ * 5 : 0, MET = GEN ? TJ * 9 : 0;
  static constexpr int STAGE = REC + DQ + MET;
  static constexpr int WORDS = TI * R * (STAGE + 5 * TJ + 8) + R * 5 * TJ;   // (x slots of one more row)
  static constexpr int SMEM = WORDS * (int)sizeof(T);
  static_assert(32 % TI == 0, "helper lanes per row");
  // a producer that takes every n-th step must not run two uses of a slot
  // ahead of the row (the parity of a phase would be ambiguous): n <= R
  static_assert(SWEEP_XH <= R && QY <= R && R % 2 == 0, "ring depth");
  static_assert(SMEM + 8 * (TI + 2) * R * 2 + 64 <= 227 * 1024, "shared memory of a pass");
};

template <class Met, bool BACKWARD, typename T>
__global__ void __launch_bounds__(SweepShape<T, !Met::kChannel, BACKWARD>::THREADS, 1)
    k_sweep(Dev d, SweepArgs a, int last) {
  using G = SweepShape<T, !Met::kChannel, BACKWARD>;
  constexpr int TI = G::TI, TJ = G::TJ, R = G::R, XH = SWEEP_XH, QY = G::QY;
  extern __shared__ __align__(128) unsigned char s_dyn[];
  T *const s_rec = reinterpret_cast<T *>(s_dyn);             // [TI][R][STAGE]
  T *const s_x = s_rec + TI * R * G::STAGE;                  // [TI + 1][R][5][TJ]
  T *const s_y = s_x + (TI + 1) * R * 5 * TJ;                // [TI][R][8]
  // per row and slot: the step's x (and y) products are posted; the row is
  // done with them.  Row TI is the sender, so that all rows run the same
  // instructions.  b_room: the next CTA of the cluster is done with the slot
  // of its first row
  __shared__ __align__(8) uint64_t b_in[TI + 1][R], b_done[TI + 1][R], b_room[R];
  __shared__ int s_ticket, s_dead, s_never;   // (s_never stays 0)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nti = (d.nx + TI - 1) / TI, ntj = (d.ny + TJ - 1) / TJ;
  // one ticket per cluster of consecutive x tiles, taken by its first CTA
  const int cx = (int)tc::cluster_nctarank(), rank = (int)tc::cluster_ctarank();
  const int units = (nti + cx - 1) / cx * ntj;
  if (threadIdx.x == 0) {
    s_dead = s_never = 0;
    if (rank == 0) s_ticket = (int)atomicAdd(a.ticket + (BACKWARD ? 1 : 0), 1u);
  }
  tc::cluster_sync();
  const int ticket = (int)tc::ld_cluster_u32(tc::mapa(tc::smem_addr(&s_ticket), 0));
  const int unit = a.order[BACKWARD ? units - 1 - ticket : ticket];
  const int ta = unit / ntj * cx + rank, tb = unit % ntj;
  const int Nz = d.nz, S = sweep_steps(d);
  const int ni = min(TI, d.nx - ta * TI), nj = min(TJ, d.ny - tb * TJ);   // rows and columns with cells
  const int Se = Nz + nj - 1;                                              // steps of a row
  const int pa = BACKWARD ? ta + 1 : ta - 1, pb = BACKWARD ? tb + 1 : tb - 1;
  const bool halo = BACKWARD ? ta == nti - 1 : ta == 0;                    // the x products are the periodic halo's
  const bool from_y = BACKWARD ? tb + 1 < ntj : tb > 0;
  // x products from / to the neighbouring CTA of the cluster
  const bool pushed = !halo && (BACKWARD ? rank + 1 < cx : rank > 0);
  const bool push = BACKWARD ? rank > 0 : rank + 1 < cx && ta + 1 < nti;
  const int row0 = BACKWARD ? ni - 1 : 0;                                  // first row of the flow
  const int polls = a.spin_limit > (1 << 28) ? 0x7fffffff : 4 * a.spin_limit + 4096;
  constexpr uint32_t PUSH_B = 5 * TJ * sizeof(T);
  T *const xbuf = a.buf<T>(a.xbuf), *const ybuf = a.buf<T>(a.ybuf);
  if (threadIdx.x < TI * R) {
    const int w = threadIdx.x / R, r = threadIdx.x % R;
    tc::mbar_init(tc::smem_addr(&b_in[w][r]), from_y ? 2 : 1);
    tc::mbar_init(tc::smem_addr(&b_done[w][r]), 1);
    if (w == 0) {
      tc::mbar_init(tc::smem_addr(&b_in[TI][r]), 1);
      tc::mbar_init(tc::smem_addr(&b_done[TI][r]), 1);
      tc::mbar_init(tc::smem_addr(&b_room[r]), 1);
    }
    // pushed products count their bytes on the slot; the row arms it
    if (pushed && w == row0 && r < Se) tc::mbar_expect_tx(tc::smem_addr(&b_in[w][r]), PUSH_B);
  }
  tc::mbar_fence_init();
  tc::cluster_sync();
  if (ta >= nti) return;

  if (warp == TI + XH + 1) {
    // ---- y helper: lane (row w, q) posts the receiving lane's values of
    // the row's steps q, q + QY, ...; the steps past its last cell are empty
    if (!from_y) return;
    const int w = lane / (32 / TI), q = lane % (32 / TI);
    int r = q, idle = 0;
    T *const src = ybuf + ((long long)(ta * TI + w) * ntj + pb) * Nz * 5;
    const bool mine = w < ni && q < QY;
    while (__any_sync(0xffffffffu, mine && r < Se)) {
      bool posted = false;
      if (mine && r < Se) {
        T *const p = src + (long long)(BACKWARD ? Nz - 1 - r : r) * 5;
        T v5[5];
        bool ok = true;
        if (r < Nz)
#pragma unroll
          for (int v = 0; v < 5; v++) {
            v5[v] = ld_gpu(p + v);
            ok = ok && !is_sentinel(v5[v]);
          }
        const bool gone = !ok && (*(volatile int *)&s_dead || (idle % 16 == 15 && given_up(&s_dead, d.status)));
        // (once the CTA has given up, its rows no longer wait, and neither
        // does this; but a row with pushed products goes on waiting, and its
        // slots, which count bytes, must not be posted ahead of it)
        const bool room = r < R || tc::mbar_test(tc::smem_addr(&b_done[w][r % R]), ((r / R) - 1) & 1) ||
                          (*(volatile int *)&s_dead && !(pushed && w == row0));
        if ((ok || gone) && room) {
          if (r < Nz) {
            T *const dst = s_y + (w * R + r % R) * 8;
#pragma unroll
            for (int v = 0; v < 5; v++) {
              dst[v] = v5[v];
              if (ok) put_sentinel(p + v);
            }
          }
          tc::mbar_arrive(tc::smem_addr(&b_in[w][r % R]));
          r += QY;
          idle = 0;
          posted = true;
        } else if (!ok) {
          // (room is awaited without a count: the row empties its slots as
          // long as its other inputs come, whose waits are counted)
          if (idle++ >= a.spin_limit) give_up(&s_dead, d.status);
        }
      }
      if (!__any_sync(0xffffffffu, posted)) __nanosleep(20);
    }
    return;
  }
  if (warp == TI + XH) {
    // ---- sender: the last row's x products, to the next CTA of the cluster
    // (pushed into its first row's slots, every lane's, so that the bytes
    // are always the same), to the next cluster's through the global buffer,
    // or (the end of the slab) nowhere
    const bool send = !push && (BACKWARD ? ta > 0 : ta + 1 < nti);
    const int up = BACKWARD ? rank - 1 : rank + 1, up_row0 = BACKWARD ? TI - 1 : 0;   // (backward, it is a whole CTA)
    const uint32_t to = push ? tc::mapa(tc::smem_addr(s_x + up_row0 * R * 5 * TJ + lane), up) : 0,
                   to_bar = push ? tc::mapa(tc::smem_addr(&b_in[up_row0][0]), up) : 0;
    T *const out = xbuf + ((long long)ta * ntj + tb) * S * (5 * TJ) + lane;
    for (int s = 0; s < Se; s++) {
      const int u = s % R;
      const uint32_t ph = (s / R) & 1;
      push_wait(tc::smem_addr(&b_in[TI][u]), ph, &s_dead, d.status);
      T v5[5];
#pragma unroll
      for (int v = 0; v < 5; v++) v5[v] = s_x[(TI * R + u) * (5 * TJ) + v * TJ + lane];
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tc::smem_addr(&b_done[TI][u]));
      if (push) {
        if (s >= R) push_wait(tc::smem_addr(&b_room[u]), ph ^ 1, &s_dead, d.status);
#pragma unroll
        for (int v = 0; v < 5; v++) tc::st_async(to + (u * 5 + v) * (uint32_t)(TJ * sizeof(T)), v5[v], to_bar + 8 * u);
      } else if (send) {
        const int sf = BACKWARD ? Se - 1 - s : s, k = sf - lane;
        if (lane < nj && k >= 0 && k < Nz)
#pragma unroll
          for (int v = 0; v < 5; v++) __stcg(out + (long long)sf * (5 * TJ) + v * TJ, v5[v]);
      }
    }
    if (cx > 1) tc::cluster_sync();
    return;
  }
  if (warp == TI && pushed) {
    // ---- receiver: arms the first row's slots for the products pushed into
    // them and returns the room
    if (lane == 0) {
      const uint32_t room = tc::mapa(tc::smem_addr(&b_room[0]), BACKWARD ? rank + 1 : rank - 1);
      for (int s = 0; s + R < Se; s++) {
        const int u = s % R;
        push_wait(tc::smem_addr(&b_done[row0][u]), (s / R) & 1, &s_dead, d.status);
        tc::mbar_expect_tx(tc::smem_addr(&b_in[row0][u]), PUSH_B);
        tc::mbar_arrive_cluster_relaxed(room + 8 * u);
      }
    }
    __syncwarp();
    tc::cluster_sync();
    return;
  }
  if (warp >= TI) {
    // ---- x helper: every XH-th step of the first row's x products
    if (pushed) return;
    T *const src = halo ? a.buf<T>(a.hx[BACKWARD]) + (long long)tb * S * (5 * TJ)
                        : xbuf + ((long long)pa * ntj + tb) * S * (5 * TJ);
    const int h = warp - TI;
    bool active = false;
    T v5[5] = {0, 0, 0, 0, 0};
    auto fetch = [&](int s) {   // the lanes' values of step s, as they are now
      const int k = (BACKWARD ? Se - 1 - s : s) - lane;
      active = lane < nj && k >= 0 && k < Nz;
      if (active)
#pragma unroll
        for (int v = 0; v < 5; v++) v5[v] = ld_gpu(src + (long long)(BACKWARD ? Se - 1 - s : s) * (5 * TJ) + v * TJ + lane);
    };
    auto missing = [&]() {
      bool m = false;
#pragma unroll
      for (int v = 0; v < 5; v++) m = m || is_sentinel(v5[v]);
      return active && !halo && m;
    };
    if (h < Se) fetch(h);
    for (int s = h; s < Se; s += XH) {
      for (int it = 0; __any_sync(0xffffffffu, missing()); it++) {
        if (it >= a.spin_limit || (it % 16 == 15 && given_up(&s_dead, d.status))) {
          if (lane == 0) give_up(&s_dead, d.status);
          break;
        }
        fetch(s);
      }
      if (s >= R) ring_wait(tc::smem_addr(&b_done[row0][s % R]), ((s / R) - 1) & 1, polls, &s_dead, d.status);
      T *const dst = s_x + (row0 * R + s % R) * (5 * TJ) + lane;
#pragma unroll
      for (int v = 0; v < 5; v++) dst[v * TJ] = v5[v];
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tc::smem_addr(&b_in[row0][s % R]));
      if (active && !halo && !missing())
#pragma unroll
        for (int v = 0; v < 5; v++) put_sentinel(src + (long long)(BACKWARD ? Se - 1 - s : s) * (5 * TJ) + v * TJ + lane);
      if (s + XH < Se) fetch(s + XH);   // under way while the other helpers post
    }
    return;
  }
  // ---- a row.  Its step is the serial chain of the pass, so it is kept to
  // one wait for the products, the arithmetic, one store of the products and
  // one arrival instruction (lane 0 on the receiving row's slot, lane 1 on
  // its own); the records come by the lanes' own asynchronous copies, R steps
  // ahead.  The loop is unrolled by the ring depth, so that every slot is a
  // compile-time offset, and a group of steps in which every lane has a cell
  // runs without the tests that the ramps need: at one warp per scheduler a
  // branch costs as much as several arithmetic instructions.
  const int w = warp;
  if (w >= ni) return;
  const int i = 3 + ta * TI + w, j = 2 + tb * TJ + lane, ie = d.nx + 2;
  const bool next_row = BACKWARD ? w > 0 : w + 1 < ni;
  const int dst_w = next_row ? (BACKWARD ? w - 1 : w + 1) : TI;     // the row that receives this row's x products
  // what lets a wait end early: the dead flag; but not for slots that count
  // pushed bytes, and not ahead of the sender (see push_wait)
  volatile int *const dead_in = pushed && w == row0 ? &s_never : &s_dead;
  volatile int *const dead_out = next_row ? &s_dead : &s_never;
  const int polls_in = pushed && w == row0 ? PUSH_POLLS : polls, polls_out = next_row ? polls : PUSH_POLLS;
  const bool y_out = BACKWARD ? tb > 0 : tb + 1 < ntj;
  const int recv_lane = BACKWARD ? nj - 1 : 0, send_lane = BACKWARD ? 0 : TJ - 1;
  // the lane that holds this lane's j neighbour; the edge lane's neighbour is
  // the wall ghost row (dQ = 0: weight 0) unless the y helper posts one
  const int src_lane = lane == recv_lane ? lane : (BACKWARD ? min(lane + 1, TJ - 1) : max(lane - 1, 0));
  const T rdx = (T)d.rdxi, rdz = (T)d.rdzt, rdt = (T)(1.0 / d.dt);
  const T rdy = lane == recv_lane && !from_y ? (T)0 : (T)d.rdet;
  const bool column = lane < nj;
  const T et = Met::kChannel && column ? (T)a.etdytab[j] : (T)1;
  const long long stream = (long long)(i - 3) * ntj + tb;
  // the block of step s is sf = s or Se - 1 - s
  constexpr int DIR = BACKWARD ? -1 : 1;
  const int sf0 = BACKWARD ? Se - 1 : 0;
  // dQ out: into the row's stream, or (first backward pass) only planes ie
  // and 3, the lagged halos of the second sweep's passes (an open slab's stay
  // zero)
  const bool to_halo = BACKWARD && !last;
  const bool store = !to_halo || (!d.x_open && (i == ie || i == 3));
  T *dq = (to_halo ? a.buf<T>(a.halo[i == ie ? 0 : 1]) + (long long)tb * S * (5 * TJ)
                   : a.buf<T>(a.dq) + stream * S * (5 * TJ)) + (long long)sf0 * (5 * TJ) + lane;
  T *const yout = ybuf + (stream * Nz + (BACKWARD ? Nz - 1 : 0)) * 5;
  const T *const x_in = s_x + w * R * 5 * TJ + lane;
  T *const x_out = s_x + dst_w * R * 5 * TJ + lane;
  const T *const y_in = s_y + w * R * 8;
  const T *const rec_in = s_rec + w * R * G::STAGE;
  const uint32_t bar_in = tc::smem_addr(&b_in[w][0]), bar_dst = tc::smem_addr(&b_done[dst_w][0]),
                 bar_arrive = lane == 0 ? tc::smem_addr(&b_in[dst_w][0]) : tc::smem_addr(&b_done[w][0]);
  // the copies of a step into its stage, one group: this lane's 16 bytes of
  // every 512 of the step's blocks
  constexpr int REC_B = G::REC * sizeof(T), DQ_B = 5 * TJ * sizeof(T), MET_B = 9 * TJ * sizeof(T);
  const char *rec_src = (const char *)(a.buf<T>(a.cellrec) + stream * S * G::REC) + (long long)sf0 * REC_B + lane * 16;
  const char *dq_src = (const char *)(a.buf<T>(a.dq) + stream * S * (5 * TJ)) + (long long)sf0 * DQ_B + lane * 16;
  const char *met_src = nullptr;
  if (!Met::kChannel) met_src = (const char *)(a.buf<T>(a.met) + stream * S * (9 * TJ)) + (long long)sf0 * MET_B + lane * 16;
  const uint32_t stage0 = tc::smem_addr(rec_in) + lane * 16;
  auto copy = [&](auto steady, int s, int stage) {   // called for s = 0, 1, 2, ...
    if (decltype(steady)::value || s < Se) {
      const uint32_t to = stage0 + stage * (uint32_t)(G::STAGE * sizeof(T));
      if (decltype(steady)::value) {
#pragma unroll
        for (int o = 0; o < REC_B; o += 512) cp_async16(to + o, rec_src + o);
      } else {
        const int sf = BACKWARD ? Se - 1 - s : s, l0 = max(0, sf - Nz + 1), l1 = min(nj - 1, sf);   // lanes with a cell
#pragma unroll
        for (int o = 0; o < REC_B; o += 512) {
          const int l = (o + lane * 16) / (int)(CR_N * sizeof(T));
          if (l >= l0 && l <= l1) cp_async16(to + o, rec_src + o);
        }
      }
      if (BACKWARD)
#pragma unroll
        for (int o = 0; o < DQ_B; o += 512)
          if (o + 512 <= DQ_B || o + lane * 16 < DQ_B) cp_async16(to + REC_B + o, dq_src + o);
      if (!Met::kChannel)
#pragma unroll
        for (int o = 0; o < MET_B; o += 512)
          if (o + 512 <= MET_B || o + lane * 16 < MET_B)
            cp_async16(to + G::DQ * (uint32_t)sizeof(T) + REC_B + o, met_src + o);
      rec_src += DIR * REC_B;
      if (BACKWARD) dq_src += DIR * DQ_B;
      if (!Met::kChannel) met_src += DIR * MET_B;
    }
    cp_async_commit();
  };
  T rec[REC_N], mr[5], mm[Met::kChannel ? 1 : 9];
  auto load = [&](int stage) {   // the oldest step under way, into registers
    cp_async_wait<R - 1>();
    __syncwarp();
    const T *const st = rec_in + stage * G::STAGE;
    load_cellrec(st + lane * CR_N, lane, rec, BACKWARD ? (T *)nullptr : mr);
    if (BACKWARD)
#pragma unroll
      for (int v = 0; v < 5; v++) mr[v] = st[G::REC + v * TJ + lane];
    if (!Met::kChannel)
#pragma unroll
      for (int v = 0; v < 9; v++) mm[v] = st[G::REC + G::DQ + v * TJ + lane];
  };
#pragma unroll
  for (int u = 0; u < R; u++) copy(std::false_type(), u, u);
  load(0);
  T ty[5] = {0, 0, 0, 0, 0}, cz[5] = {0, 0, 0, 0, 0};
  int kf = BACKWARD ? lane - (nj - 1) : -lane;    // the lane's cell, counted in the order of the pass
  uint32_t parity = 0;                            // of the slots' current use
  // one step; `steady`: every column has a cell at this step and R steps on
  auto step = [&](auto steady, int s, int u) {
    constexpr bool STEADY = decltype(steady)::value;
    // lanes without a cell carry arbitrary values along, which reach no lane
    // with a cell: an i, j or k neighbour without a cell is masked here or at
    // the lane's edge
    const bool active = STEADY ? column : column && (unsigned)kf < (unsigned)Nz;
    ring_wait(bar_in + 8 * u, parity, polls_in, dead_in, d.status);
    T tx[5];
#pragma unroll
    for (int v = 0; v < 5; v++) tx[v] = x_in[(u * 5 + v) * TJ];
    if (from_y && lane == recv_lane)
#pragma unroll
      for (int v = 0; v < 5; v++) ty[v] = y_in[u * 8 + v];
    if (!STEADY && kf == 0)   // its z neighbour is the ghost row: dQ = 0
#pragma unroll
      for (int v = 0; v < 5; v++) cz[v] = (T)0;
    T L[5];
#pragma unroll
    for (int v = 0; v < 5; v++) L[v] = fma_rn(cz[v], rdz, fma_rn(tx[v], rdx, mul_rn(ty[v], rdy)));
    const T d11 = rec[R_D11], d22 = rec[R_D22], d51 = rec_d51<T>(rec, rdt);
    T n[5];
    if (!BACKWARD) {
      // Dual_time_stepping.cpp:1289-1293
      T r1 = mr[0] - L[0];
      n[0] = d11 * r1;
      n[1] = d22 * (mr[1] - L[1]);
      n[2] = d22 * (mr[2] - L[2]);
      n[3] = d22 * (mr[3] - L[3]);
      n[4] = fma_rn(d22, mr[4] - L[4], mul_rn(d51, r1));
    } else {
      // Dual_time_stepping.cpp:1651-1655 (mr holds this cell's forward result)
      n[0] = fma_rn(-d11, L[0], mr[0]);
      n[1] = fma_rn(-d22, L[1], mr[1]);
      n[2] = fma_rn(-d22, L[2], mr[2]);
      n[3] = fma_rn(-d22, L[3], mr[3]);
      n[4] = mr[4] - fma_rn(d22, L[4], mul_rn(d51, L[0]));
    }
    T ox[5], oy[5];
    if (Met::kChannel) {
      // the channel's face metrics have one nonzero component per direction
      // (1, etdy, 1 on the x, y, z components), so only the nonzero split
      // entries are formed and applied
      channel_products<T, 0, BACKWARD>(rec, (T)1, n, ox);
      channel_products<T, 1, BACKWARD>(rec, et, n, oy);
      channel_products<T, 2, BACKWARD>(rec, (T)1, n, cz);
    } else {
      const Split<T> Ax = split_from_record<T>(rec, 0, mm[0], mm[1], mm[2]);
      const Split<T> Ay = split_from_record<T>(rec, 1, mm[3], mm[4], mm[5]);
      const Split<T> Az = split_from_record<T>(rec, 2, mm[6], mm[7], mm[8]);
      if (BACKWARD) {
        upper_terms<T>(Ax, n, ox);
        upper_terms<T>(Ay, n, oy);
        upper_terms<T>(Az, n, cz);
      } else {
        lower_terms<T>(Ax, n, ox);
        lower_terms<T>(Ay, n, oy);
        lower_terms<T>(Az, n, cz);
      }
    }
    // hand the x products on (room is awaited for two steps at a time)
    if (u % 2 == 0 && (STEADY || s + 1 >= R))
      ring_wait(bar_dst + 8 * (u + 1), parity ^ 1, polls_out, dead_out, d.status);
#pragma unroll
    for (int v = 0; v < 5; v++) x_out[(u * 5 + v) * TJ] = ox[v];
    __syncwarp();
    // every lane has read its inputs and written its products
    if (lane < 2) tc::mbar_arrive(bar_arrive + 8 * u);
#pragma unroll
    for (int v = 0; v < 5; v++) ty[v] = __shfl_sync(0xffffffffu, oy[v], src_lane);
    copy(steady, s + R, u);
    if (store && active)
#pragma unroll
      for (int v = 0; v < 5; v++) dq[v * TJ] = n[v];
    if (y_out && lane == send_lane && active)
#pragma unroll
      for (int v = 0; v < 5; v++) __stcg(yout + DIR * 5 * kf + v, oy[v]);
    dq += DIR * 5 * TJ;
    kf++;
    if (STEADY || s + 1 < Se) load((u + 1) % R);
  };
  for (int s0 = 0; s0 < Se; s0 += R, parity ^= 1) {
    if (s0 >= max(nj, R) && s0 + 2 * R <= Nz) {
#pragma unroll
      for (int u = 0; u < R; u++) step(std::true_type(), s0 + u, u);
    } else {
#pragma unroll
      for (int u = 0; u < R; u++)
        if (s0 + u < Se) step(std::false_type(), s0 + u, u);
    }
  }
  // a CTA stays until its neighbours have sent it their last signals
  if (cx > 1) tc::cluster_sync();
}

// Dual_time_stepping.cpp:1702-1743 after the last backward pass: the
// primitive update of every interior cell from its final dQ (read from the
// rows' streams), fully parallel rather than inside the wavefront's chain of
// dependent steps, with per-block partial sums of the squared increments
// (:1761-1776).  The divisions by q1, rho, T and J are Newton-refined
// reciprocals (1/J from the table).
//
// A block owns UPD_TJ columns of one row and UPD_KC consecutive k of them.
// In the row's stream those cells lie in UPD_KC + UPD_TJ - 1 consecutive
// steps, each holding the columns' values side by side: the block reads them
// whole into shared memory, then each warp updates 32 consecutive k of one
// column, so the reads and writes of the state in the reference layout are
// coalesced too.
constexpr int UPD_KC = 32, UPD_TJ = 16;
inline unsigned sweep_update_grid_x(const Dev &d) { return (unsigned)(d.nx * ((d.ny + UPD_TJ - 1) / UPD_TJ)); }
inline unsigned sweep_update_grid_y(const Dev &d) { return (unsigned)((d.nz + UPD_KC - 1) / UPD_KC); }

template <typename T>
__global__ void __launch_bounds__(256) k_update_skewed(Dev d, SweepArgs a) {
  constexpr int NS = UPD_KC + UPD_TJ - 1;   // steps holding the block's cells
  static_assert(SWEEP_TJ % UPD_TJ == 0 && UPD_TJ == 16, "column staging; two rows per warp");
  __shared__ T sdq[5][NS][UPD_TJ + 1];       // (+1: the update reads a column down the steps)
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) a.clock[1] = globaltimer();
  const int status = *(volatile int *)d.status;
  const int ntu = (d.ny + UPD_TJ - 1) / UPD_TJ, S = sweep_steps(d);
  const int row = blockIdx.x / ntu, j0 = blockIdx.x % ntu * UPD_TJ;   // 0-based row and first column
  const int ntj = (d.ny + SWEEP_TJ - 1) / SWEEP_TJ, l0 = j0 % SWEEP_TJ;
  const int k0 = blockIdx.y * UPD_KC;        // first k of the block (0-based)
  const int s0 = k0 + l0;                    // step of the cell (first column, k0)
  const T *const dq = a.buf<T>(a.dq) + ((long long)row * ntj + j0 / SWEEP_TJ) * S * (5 * SWEEP_TJ) + l0;
  // the warp's two rows of the state, in flight while dQ is staged
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = 3 + row, kl = k0 + lane;
  double q[2][5], Jc[2], iJc[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int j = 2 + j0 + warp + 8 * h;
    if (j > d.ny + 1 || kl >= d.nz) continue;
    const long long c = ix(d, i, j, 2 + kl), cj = a.channel_metrics ? ix(d, 3, j, 2) : c;
#pragma unroll
    for (int v = 0; v < 5; v++) q[h][v] = d.U_[v][c];
    Jc[h] = d.J[cj];
    iJc[h] = d.iJ[cj];
  }
  for (int e = threadIdx.x; e < NS * UPD_TJ; e += blockDim.x) {
    const int ls = e / UPD_TJ, jl = e % UPD_TJ, st = s0 + ls;
    if (st < S) {
#pragma unroll
      for (int v = 0; v < 5; v++) sdq[v][ls][jl] = dq[(long long)st * (5 * SWEEP_TJ) + v * SWEEP_TJ + jl];
    }
  }
  // a wavefront pass that gave up left dQ incomplete: keep the state
  if (status) return;
  __syncthreads();
  double acc[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int jl = warp + 8 * h, j = 2 + j0 + jl;
    if (j > d.ny + 1 || kl >= d.nz) continue;
    const int ls = lane + jl;            // step of the cell, relative to s0
    const long long c = ix(d, i, j, 2 + kl);
    const double J = Jc[h], iJ = iJc[h];
    const double q1 = q[h][0], iq1 = nr_rcp(q1);
    const double rhoold = q1 * J;
    const double Uold = q[h][1] * iq1, Vold = q[h][2] * iq1, Wold = q[h][3] * iq1;
    const double VVold = Uold * Uold + Vold * Vold + Wold * Wold;
    const double Pold = (q[h][4] * J - 0.5 * rhoold * VVold) * (KG - 1);
    const double Told = Pold * (iq1 * iJ);   // 1 / rho = 1 / (q1 J)
    const double P = Pold + (double)sdq[0][ls][jl] * J, U = Uold + (double)sdq[1][ls][jl] * J;
    const double V = Vold + (double)sdq[2][ls][jl] * J, W = Wold + (double)sdq[3][ls][jl] * J;
    const double Tn = Told + (double)sdq[4][ls][jl] * J;
    const double rho = P * nr_rcp(Tn), rJ = rho * iJ;
    d.U_[0][c] = rJ;
    d.U_[1][c] = rJ * U;
    d.U_[2][c] = rJ * V;
    d.U_[3][c] = rJ * W;
    d.U_[4][c] = (P * (1 / (KG - 1)) + 0.5 * rho * (U * U + V * V + W * W)) * iJ;
    acc[0] += (rho - rhoold) * (rho - rhoold);
    acc[1] += (U - Uold) * (U - Uold);
    acc[2] += (V - Vold) * (V - Vold);
    acc[3] += (W - Wold) * (W - Wold);
    acc[4] += (Tn - Told) * (Tn - Told);
  }
  block_sum5(acc, d.partial + 5 * ((long long)blockIdx.y * gridDim.x + blockIdx.x));
}

template <typename T>
static void launch_update_skewed(const Dev &d, const SweepArgs &a, cudaStream_t s) {
  k_update_skewed<T><<<dim3(sweep_update_grid_x(d), sweep_update_grid_y(d)), 256, 0, s>>>(d, a);
}
int sweep_update_blocks(const Dev &d) { return (int)(sweep_update_grid_x(d) * sweep_update_grid_y(d)); }

// tickets follow the step at which the wavefront reaches a cluster, `rows`
// steps per cluster along x and 32 per column block along y
void sweep_tile_order(int ncx, int ntj, int rows, std::vector<int> &order) {
  order.resize((size_t)ncx * ntj);
  for (int t = 0; t < ncx * ntj; t++) order[t] = t;
  std::stable_sort(order.begin(), order.end(), [&](int p, int q) {
    return p / ntj * rows + p % ntj * SWEEP_TJ < q / ntj * rows + q % ntj * SWEEP_TJ;
  });
}

// CTAs per cluster along x for nti tiles: enough for all of them, at most 8,
// if the device holds such a cluster of the largest wavefront kernel
template <typename T>
static int cluster_x_for(int nti) {
  using B = SweepShape<T, true, true>;
  int cx = 1;
  while (cx < 8 && cx < nti) cx *= 2;
  for (; cx > 1; cx /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cx);
    cfg.blockDim = dim3(B::THREADS);
    cfg.dynamicSmemBytes = B::SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cx;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_sweep<MetricsGeneral, true, T>, &cfg) == cudaSuccess && n >= 1) return cx;
    cudaGetLastError();
  }
  return 1;
}
int sweep_cluster_x(int nti, bool mixed) { return mixed ? cluster_x_for<float>(nti) : cluster_x_for<double>(nti); }

template <class Met, typename T>
static void run_halo_products(const Dev &d, const SweepArgs &a, cudaStream_t s, bool first) {
  k_halo_products<Met, T><<<dim3((d.nz + 63) / 64, d.ny, 2), 64, 0, s>>>(d, a, first);
}
template <class Met, typename T>
static void run_pass(const Dev &d, const SweepArgs &a, cudaStream_t s, bool backward, bool last) {
  const int cx = a.cluster_x, ncx = (sweep_tiles_x<T>(d.nx) + cx - 1) / cx;
  using F = SweepShape<T, !Met::kChannel, false>;
  using B = SweepShape<T, !Met::kChannel, true>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncx * cx * sweep_tiles_y(d.ny));
  cfg.blockDim = dim3(F::THREADS);
  cfg.dynamicSmemBytes = backward ? B::SMEM : F::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cx;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (!backward) cudaLaunchKernelEx(&cfg, k_sweep<Met, false, T>, d, a, (int)last);
  else cudaLaunchKernelEx(&cfg, k_sweep<Met, true, T>, d, a, (int)last);
}
// one symmetric sweep; its backward dQ is stored only when the update follows
template <class Met, typename T>
static void run_sweep(const Dev &d, const SweepArgs &a, cudaStream_t s, bool last) {
  run_halo_products<Met, T>(d, a, s, !last);
  run_pass<Met, T>(d, a, s, false, last);
  run_pass<Met, T>(d, a, s, true, last);
}

#define SWEEP_DISPATCH(fn, ...)                                        \
  do {                                                                 \
    if (mixed) {                                                       \
      if (a.channel_metrics) fn<MetricsChannel, float>(__VA_ARGS__);   \
      else fn<MetricsGeneral, float>(__VA_ARGS__);                     \
    } else {                                                           \
      if (a.channel_metrics) fn<MetricsChannel, double>(__VA_ARGS__);  \
      else fn<MetricsGeneral, double>(__VA_ARGS__);                    \
    }                                                                  \
  } while (0)

void launch_sweep_pass(const Dev &d, const SweepArgs &a, cudaStream_t s, bool mixed, bool backward, bool last) {
  if (!backward) SWEEP_DISPATCH(run_halo_products, d, a, s, !last);
  SWEEP_DISPATCH(run_pass, d, a, s, backward, last);
}

void launch_sweep_update(const Dev &d, const SweepArgs &a, cudaStream_t s, bool mixed) {
  if (mixed) launch_update_skewed<float>(d, a, s);
  else launch_update_skewed<double>(d, a, s);
}

void launch_sweeps(const Dev &d, const SweepArgs &a, cudaStream_t s, bool mixed) {
  for (int sweep = 0; sweep < 2; sweep++) SWEEP_DISPATCH(run_sweep, d, a, s, sweep == 1);
}

// the wavefront kernels' rings exceed 48 KB: opt in once, outside any capture
template <class Met, typename T>
static cudaError_t opt_in() {
  cudaError_t e = cudaFuncSetAttribute(k_sweep<Met, false, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       SweepShape<T, !Met::kChannel, false>::SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sweep<Met, true, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             SweepShape<T, !Met::kChannel, true>::SMEM);
  return e;
}
cudaError_t sweep_kernel_attributes() {
  cudaError_t e = opt_in<MetricsChannel, double>();
  if (e == cudaSuccess) e = opt_in<MetricsGeneral, double>();
  if (e == cudaSuccess) e = opt_in<MetricsChannel, float>();
  if (e == cudaSuccess) e = opt_in<MetricsGeneral, float>();
  return e;
}

}  // namespace cgli
